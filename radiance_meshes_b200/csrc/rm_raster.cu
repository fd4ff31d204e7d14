// Stages 5-6 on the GPU: per-pixel front-to-back integration of the tile lists
// and its reverse pass.
//
// Reference behaviour reproduced: slang/alphablend_shader_interp.slang:83-431
// (pixel state, distortion moments, forward loop with early termination at
// log-transmittance < -5.5, backward replay with state undo),
// slang/interp_version.slang:21-153 (closed-form segment integral of constant
// density and linear colour), slang/intersect.slang:393-624 (ray/tet slab
// test), slang/camera.slang:241-346 (ray generation).
//
// Design (not the reference's structure):
//   * Tets are packed once per frame into 128-byte records: the four outward
//     face planes relative to the CAMERA POSITION (n_i, D_i), the colour field
//     folded to (grd, s0 = grd.(cam - v0), base, density) - 96 bytes that are
//     staged in shared memory - and the edge lines of the tet's projected hull
//     (32 bytes, read only to decide whether a tet can touch a tile's samples).
//     The per-pixel origin offset o = cam + min_t*d only shifts each plane
//     distance by min_t*(n_i.d), so the per-(pixel,tet) work drops from four
//     cross products to four dot products.
//   * 16 pixels of one tile are a unit, walked by a half-warp or, two lanes per
//     pixel, by a warp.  Forward: the list is examined one entry per lane
//     (hull lines against the box of the unit's samples); survivors are
//     tested against each of the 16 sample positions, which gives the mask of
//     pixels a tet can cover; entries with a non-empty mask are staged in batches
//     with 128-bit cp.async copies that land while the next ones are examined, and
//     every lane then walks only the staged entries that cover its pixel.  A unit
//     stops as soon as all of its pixels have terminated.  Every evaluated batch is
//     appended, with the per-pixel bit sets of the entries that were hit, to the
//     unit's hit list.
//   * Backward walks the hit lists back to front: a lane per pixel evaluates the hits
//     and reduces each to seven scalars, then a lane per entry sums them over the 16
//     pixels into a per-tet row of record gradients; a per-tet kernel applies the chain
//     rule to vertices and cell values (12 vertex atomics per tet instead of 19 atomics
//     per pixel hit).

#include <type_traits>

#include <algorithm>
#include <climits>

#include "rm_common.cuh"

namespace rm {

// Record of a tet: 6 float4 that the integration kernels stage (four planes in pairs, colour field, base colour and
// density) and 2 with the hull lines.  A record fills 32-byte sectors of its own: tets 2k and 2k + 1 share 288 bytes and
// leave the last 32 of them unused, so that no write is a partial sector, which L2 would first fetch from DRAM.
__device__ __forceinline__ int64_t record_at(int64_t tet) { return 9 * tet - (tet & 1); }  // in float4
constexpr int kLinesAt = 6;
static_assert(RM_RECORD_FLOATS == 36, "two records and a gap fill twice this");

// ----------------------------------------------------------------------------
// Record packing
// ----------------------------------------------------------------------------
struct PlaneSetup {
  f3 n[4];
  float D[4];
  float sgn[4];
};

// Hull lines.  A ray can only hit a tet if it passes through the convex hull of the tet's central projection onto the
// plane z = 1 in front of the camera, here in pixels of an undistorted pinhole with the camera's K; a sample is where the
// ray of a pixel, whatever its lens, meets that plane.  Four lines a x + b y + c >= 0 inside, (a, b) a unit normal in
// 16-bit steps of 1/32767 (so all three in units of that) and c then chosen so that all four vertices are inside: rounding
// turns a line by at most 2e-5, which costs an edge of a hundred pixels a five-hundredth of a pixel.  8 bytes per line, 32
// per tet: one sector.
constexpr float kLineUnit = 32767.0f;
constexpr float kPixelMargin = 0.01f * kLineUnit;    // a sample up to a hundredth of a pixel outside a line is still tested
constexpr float kFisheyeMargin = 0.05f * kLineUnit;  // the same for a fisheye, whose rays far off the axis project less exactly
struct HullLines {
  float a[4], b[4], c[4];
};
__device__ __forceinline__ float pack_normal(float x, float y) {  // each with an offset of 32768, x in the low half
  return __uint_as_float((unsigned)(__float2int_rn(x * kLineUnit) + 32768) |
                         (unsigned)(__float2int_rn(y * kLineUnit) + 32768) << 16);
}
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
  float2 r;
  asm("add.rn.f32x2 %0, %1, %2;"
      : "=l"(reinterpret_cast<unsigned long long&>(r))
      : "l"(reinterpret_cast<unsigned long long&>(a)), "l"(reinterpret_cast<unsigned long long&>(b)));
  return r;
}
__device__ __forceinline__ float2 unpack_normal(float f) {
  // 2^23 + u is a float whose low mantissa bits are u
  const unsigned u = __float_as_uint(f);
  return add2(make_float2(__uint_as_float(__byte_perm(u, 0x4B000000u, 0x7410)), __uint_as_float(__byte_perm(u, 0x4B000000u, 0x7432))),
              make_float2(-8421376.0f, -8421376.0f));
}
__device__ __forceinline__ HullLines unpack_lines(float4 l0, float4 l1) {
  const float2 p0 = unpack_normal(l0.x), p1 = unpack_normal(l0.z), p2 = unpack_normal(l1.x), p3 = unpack_normal(l1.z);
  return {{p0.x, p1.x, p2.x, p3.x}, {p0.y, p1.y, p2.y, p3.y}, {l0.y, l0.w, l1.y, l1.w}};
}
// c of the first line of a tet that no ray can hit (density zero, or not a tet): the line separates every box
__device__ __forceinline__ float never_seen() { return __int_as_float(0xff800000); }

// Products with the contraction spelled out: rays that graze a tet are decided by the last bits of its planes, and these
// keep the decisions from changing with the code around them.
__device__ __forceinline__ float dot_fma(f3 a, f3 b) { return fmaf(a.z, b.z, fmaf(a.x, b.x, __fmul_rn(a.y, b.y))); }
__device__ __forceinline__ f3 cross_fma(f3 a, f3 b) {
  return {fmaf(a.y, b.z, -__fmul_rn(a.z, b.y)), fmaf(a.z, b.x, -__fmul_rn(a.x, b.z)), fmaf(a.x, b.y, -__fmul_rn(a.y, b.x))};
}

__device__ __forceinline__ void make_planes(const f3 v[4], f3 cam, PlaneSetup& p) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    // faces (v0,v1,v2) (v0,v1,v3) (v0,v2,v3) (v1,v2,v3); opposite vertex v3 v2 v1 v0
    const int b = i == 3 ? 1 : 0;
    const int e1 = i < 2 ? 1 : 2;
    const int e2 = i == 0 ? 2 : 3;
    const int op = 3 - i;
    f3 n = cross_fma(v[e1] - v[b], v[e2] - v[b]);
    float s = 1.0f;
    if (dot_fma(n, v[op] - v[b]) > 0.0f) {
      n = -n;
      s = -1.0f;
    }
    p.n[i] = n;
    p.sgn[i] = s;
    p.D[i] = -dot_fma(n, v[b] - cam);
  }
}

constexpr int kPackThreads = 128;

// Record of tet g, whose vertices are `id`.
__device__ __forceinline__ void build_record(float4* r, int4 id, const float* __restrict__ vertices, const float* __restrict__ cell,
                                             int64_t g, float density, const RmCamera& rcam) {
  f3 cam = {__ldg(rcam.cam_pos), __ldg(rcam.cam_pos + 1), __ldg(rcam.cam_pos + 2)};
  f3 v[4] = {load3(vertices, id.x), load3(vertices, id.y), load3(vertices, id.z), load3(vertices, id.w)};
  PlaneSetup p;
  make_planes(v, cam, p);
  const float* c = cell + 7 * g;
  f3 base = {__ldg(c + 1), __ldg(c + 2), __ldg(c + 3)};
  f3 grd = {__ldg(c + 4), __ldg(c + 5), __ldg(c + 6)};
  float s0 = dot_fma(grd, cam - v[0]);
#pragma unroll
  for (int i = 0; i < 4; i += 2) {  // planes in pairs: operands of the packed arithmetic of the slab test
    r[i] = make_float4(p.n[i].x, p.n[i + 1].x, p.n[i].y, p.n[i + 1].y);
    r[i + 1] = make_float4(p.n[i].z, p.n[i + 1].z, -p.D[i], -p.D[i + 1]);
  }
  r[4] = make_float4(grd.x, grd.y, grd.z, s0);
  r[5] = make_float4(base.x, base.y, base.z, density);
  // Vertices in pixel coordinates.  Only meaningful with the whole tet in front of the camera; otherwise the cull is
  // disabled for this tet (NaN lines).
  const float* W = rcam.world_view_transform;
  const float fx = __ldg(rcam.K + 0), cx = __ldg(rcam.K + 2), fy = __ldg(rcam.K + 4), cy = __ldg(rcam.K + 5);
  float px[4], py[4];
  bool ok = true;
  // Bound of the fp32 rounding error of the projected vertices, in pixels: the camera-space
  // coordinates are sums of four products (error <= 4 * 2^-24 * sum of magnitudes), and the error of
  // X/Z grows with 1/Z, so vertices near the camera plane project with errors far above the 0.01
  // pixel margin of the hull tests.  The lines are moved outwards by the bound (two end points per
  // line); a tet whose bound reaches half a pixel, or with a vertex behind the near plane, is not culled.
  float perr = 0.0f;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    float X = __ldg(W + 0) * v[k].x + __ldg(W + 1) * v[k].y + __ldg(W + 2) * v[k].z + __ldg(W + 3);
    float Y = __ldg(W + 4) * v[k].x + __ldg(W + 5) * v[k].y + __ldg(W + 6) * v[k].z + __ldg(W + 7);
    float Z = __ldg(W + 8) * v[k].x + __ldg(W + 9) * v[k].y + __ldg(W + 10) * v[k].z + __ldg(W + 11);
    const float u4 = 2.4e-7f;
    const float eX = u4 * (fabsf(__ldg(W + 0) * v[k].x) + fabsf(__ldg(W + 1) * v[k].y) + fabsf(__ldg(W + 2) * v[k].z) + fabsf(__ldg(W + 3)));
    const float eY = u4 * (fabsf(__ldg(W + 4) * v[k].x) + fabsf(__ldg(W + 5) * v[k].y) + fabsf(__ldg(W + 6) * v[k].z) + fabsf(__ldg(W + 7)));
    const float eZ = u4 * (fabsf(__ldg(W + 8) * v[k].x) + fabsf(__ldg(W + 9) * v[k].y) + fabsf(__ldg(W + 10) * v[k].z) + fabsf(__ldg(W + 11)));
    ok = ok && Z > 1e-3f;
    const float iz = 1.0f / Z;
    px[k] = fx * (X * iz) + cx;
    py[k] = fy * (Y * iz) + cy;
    const float ex = fabsf(fx) * iz * (eX + fabsf(X * iz) * eZ) + 4e-7f * (fabsf(px[k]) + fabsf(cx));
    const float ey = fabsf(fy) * iz * (eY + fabsf(Y * iz) * eZ) + 4e-7f * (fabsf(py[k]) + fabsf(cy));
    perr = fmaxf(perr, ex + ey);
  }
  const float margin = 2.0f * perr;
  ok = ok && margin < 0.5f;
  // A vertex pair is a hull edge iff the other two vertices lie on one side of its line; a tet projects to a
  // quadrilateral (4 such pairs) or to a triangle with one vertex inside (3).  Anything else is degenerate and
  // disables the cull for this tet.
  float lab[4] = {0, 0, 0, 0}, lc[4] = {0, 0, 0, 0};
  int ne = 0;
#pragma unroll
  for (int a = 0; a < 4; ++a) {
#pragma unroll
    for (int b = a + 1; b < 4; ++b) {
      const int c1 = (a != 0 && b != 0) ? 0 : ((a != 1 && b != 1) ? 1 : 2);
      const int c2 = 6 - a - b - c1;
      const float nx = -(py[b] - py[a]), ny = px[b] - px[a];
      const float len2 = nx * nx + ny * ny;
      const float s1 = nx * (px[c1] - px[a]) + ny * (py[c1] - py[a]);
      const float s2 = nx * (px[c2] - px[a]) + ny * (py[c2] - py[a]);
      const bool pos = s1 >= 0.0f && s2 >= 0.0f && (s1 > 0.0f || s2 > 0.0f);
      const bool neg = s1 <= 0.0f && s2 <= 0.0f && (s1 < 0.0f || s2 < 0.0f);
      if ((pos || neg) && len2 > 0.0f) {
        const float inv = pos ? rsqrtf(len2) : -rsqrtf(len2);
        const float ab = pack_normal(nx * inv, ny * inv);
        const float2 n = unpack_normal(ab);
        const float low = fminf(fminf(n.x * px[0] + n.y * py[0], n.x * px[1] + n.y * py[1]),
                                fminf(n.x * px[2] + n.y * py[2], n.x * px[3] + n.y * py[3]));
#pragma unroll
        for (int q = 0; q < 4; ++q) {  // slot `ne`, without dynamic indexing
          if (q == ne) { lab[q] = ab; lc[q] = fmaf(margin, kLineUnit, -low); }
        }
        ++ne;
      }
    }
  }
  ok = ok && (ne == 3 || ne == 4);
  if (ne == 3) { lab[3] = lab[2]; lc[3] = lc[2]; }
  if (!ok) {
    const float qnan = __int_as_float(0x7fc00000);
#pragma unroll
    for (int k = 0; k < 4; ++k) lc[k] = qnan;
  }
  r[6] = make_float4(lab[0], lc[0], lab[1], lc[1]);
  r[7] = make_float4(lab[2], lc[2], lab[3], lc[3]);
}

// A thread builds one record in registers; it is then written through shared memory, so that the global stores are contiguous.
// What of a record is written: nothing for a culled tet, which appears in no list; the lines' sector for a tet of zero density
// (a mark), which the integration kernels drop by its first line without reading more (40 % of the tets of an unbounded scene);
// else all of it.
// PER = 1: a thread per tet.  PER > 1: the block first looks at PER tets per thread and lists those to be written whole; each of
// its warps then takes 32 of the list at a time, so that all lanes have a record to build and no warp waits for another one (of
// 6M tets 46 % have one, by runs: a list per warp leaves its last round half empty, 256 us in place of 236).
template <int PER>
__global__ void __launch_bounds__(kPackThreads, 8)
k_pack_records(const int32_t* __restrict__ indices, const float* __restrict__ vertices,
               const float* __restrict__ cell, int64_t T, int64_t V, RmCamera rcam,
               const int32_t* __restrict__ tiles_touched, float4* __restrict__ records, uint8_t* __restrict__ clear_a,
               uint8_t* __restrict__ clear_b) {
  constexpr int kRow = 9;  // 8 used; the odd stride spreads the rows over the banks
  constexpr int kTets = PER * kPackThreads;
  __shared__ __align__(16) float4 sm[kPackThreads * kRow];
  __shared__ uint16_t list[kTets];  // PER = 1: what of the thread's record is written
  __shared__ int n_listed;
  const int64_t g0 = (int64_t)blockIdx.x * kTets;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  float4* const rows = sm + 32 * warp * kRow;
  if (PER > 1 && threadIdx.x == 0) n_listed = 0;
  bool live[PER], ids_ok[PER];
  float density[PER];
  int4 id[PER];
#pragma unroll
  for (int k = 0; k < PER; ++k) {
    const int64_t g = g0 + k * kPackThreads + threadIdx.x;
    live[k] = g < T && !(tiles_touched && tiles_touched[g] == 0);
    if (g < T && clear_a) clear_a[g] = 0;
    if (g < T && clear_b) clear_b[g] = 0;
  }
#pragma unroll
  for (int k = 0; k < PER; ++k)
    density[k] = live[k] ? fmaxf(__ldg(cell + 7 * (g0 + k * kPackThreads + threadIdx.x)), 0.0f) : 0.0f;
#pragma unroll
  for (int k = 0; k < PER; ++k) {
    ids_ok[k] = false;
    if (density[k] > 0.0f) {
      // a tet that names a vertex outside the table (the projection stage culls it and reports it) is marked like one of
      // zero density: no pixel can hit it
      id[k] = __ldg(reinterpret_cast<const int4*>(indices) + g0 + k * kPackThreads + threadIdx.x);
      ids_ok[k] = (uint32_t)id[k].x < (uint64_t)V && (uint32_t)id[k].y < (uint64_t)V && (uint32_t)id[k].z < (uint64_t)V &&
                  (uint32_t)id[k].w < (uint64_t)V;
    }
  }
  if constexpr (PER == 1) {
    enum { kNone, kMark, kAll };
    const int64_t g = g0 + threadIdx.x;
    float4* r = sm + threadIdx.x * kRow;
    list[threadIdx.x] = !live[0] ? kNone : ids_ok[0] ? kAll : kMark;
    r[6] = make_float4(0.0f, never_seen(), 0.0f, 0.0f);
    r[7] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (ids_ok[0]) build_record(r, id[0], vertices, cell, g, density[0], rcam);
    __syncthreads();
    const int n_rec = (int)min((int64_t)kPackThreads, T - g0);
    for (int i = threadIdx.x; i < n_rec * 8; i += kPackThreads) {
      const int row = i >> 3, k = i & 7;
      if (list[row] == kAll || (list[row] == kMark && k >= kLinesAt)) records[record_at(g0 + row) + k] = sm[row * kRow + k];
    }
    return;
  }
  __syncthreads();
  {
    unsigned w[PER];
    int n = 0, first = 0;
#pragma unroll
    for (int k = 0; k < PER; ++k) {
      w[k] = __ballot_sync(0xffffffffu, ids_ok[k]);
      n += __popc(w[k]);
    }
    if (lane == 0 && n) first = atomicAdd(&n_listed, n);
    first = __shfl_sync(0xffffffffu, first, 0);
#pragma unroll
    for (int k = 0; k < PER; ++k) {
      if (ids_ok[k]) list[first + __popc(w[k] & ((1u << lane) - 1u))] = (uint16_t)(k * kPackThreads + threadIdx.x);
      first += __popc(w[k]);
      if (live[k] && !ids_ok[k]) {
        float4* const lines = records + record_at(g0 + k * kPackThreads + threadIdx.x) + kLinesAt;
        lines[0] = make_float4(0.0f, never_seen(), 0.0f, 0.0f);
        lines[1] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      }
    }
  }
  __syncthreads();
  const int n = n_listed;
  for (int first = 32 * warp; first < n; first += kPackThreads) {
    if (first + lane < n) {
      const int64_t g = g0 + list[first + lane];
      build_record(rows + lane * kRow, __ldg(reinterpret_cast<const int4*>(indices) + g), vertices, cell, g, __ldg(cell + 7 * g), rcam);
    }
    __syncwarp();
    const int n_rec = min(32, n - first);
    for (int i = lane; i < n_rec * 8; i += 32) {
      const int row = i >> 3, k = i & 7;
      records[record_at(g0 + list[first + row]) + k] = rows[row * kRow + k];
    }
    __syncwarp();
  }
}

// Box of the samples of a half-warp: centre, half extents, and how far outside a line it counts as missed.
struct SampleBox {
  float4 box;  // x, y, half extents
  float margin;
};
// True if one of the four hull lines of a tet has the whole box on its outer side by more than the margin.
// Conservative: NaN lines never separate.
__device__ __forceinline__ bool hull_misses_box(float4 l0, float4 l1, const SampleBox& s) {
  const HullLines h = unpack_lines(l0, l1);
  float v[4];
#pragma unroll
  for (int k = 0; k < 4; ++k)  // largest value of the line over the box
    v[k] = fmaf(fabsf(h.a[k]), s.box.z, fmaf(fabsf(h.b[k]), s.box.w, fmaf(h.a[k], s.box.x, fmaf(h.b[k], s.box.y, h.c[k]))));
  return fminf(fminf(v[0], v[1]), fminf(v[2], v[3])) < -s.margin;
}

// ----------------------------------------------------------------------------
// Ray generation (fp32), slang/camera.slang:241-346
// ----------------------------------------------------------------------------
__device__ __forceinline__ void undistort(float& px, float& py, const float* dist) {
  float k1 = dist[0], k2 = dist[1], p1 = dist[2], p2 = dist[3];
  if (k1 * k1 + k2 * k2 + p1 * p1 + p2 * p2 < 1e-9f) return;
  float x = px, y = py;
  for (int i = 0; i < 10; ++i) {
    float r2 = x * x + y * y;
    float d = 1.0f + r2 * (k1 + r2 * k2);
    float fx = d * x + 2.0f * p1 * x * y + p2 * (r2 + 2.0f * x * x) - px;
    float fy = d * y + 2.0f * p2 * x * y + p1 * (r2 + 2.0f * y * y) - py;
    float d_r = k1 + r2 * (2.0f * k2);
    float d_x = 2.0f * x * d_r;
    float d_y = 2.0f * y * d_r;
    float fx_x = d + d_x * x + 2.0f * p1 * y + 6.0f * p2 * x;
    float fx_y = d_y * x + 2.0f * p1 * x + 2.0f * p2 * y;
    float fy_x = d_x * y + 2.0f * p2 * y + 2.0f * p1 * x;
    float fy_y = d + d_y * y + 2.0f * p2 * x + 6.0f * p1 * y;
    float denom = fy_x * fx_y - fx_x * fy_y;
    if (fabsf(denom) < 1e-9f) break;
    float xn = fx * fy_y - fy * fx_y;
    float yn = fy * fx_x - fx * fy_x;
    x += xn / denom;
    y += yn / denom;
  }
  px = x;
  py = y;
}

// sample: where the ray meets the plane of the hull lines, NaN if it does not or not exactly enough for the margin
__device__ __forceinline__ f3 ray_direction(const RmCamera& c, float px, float py, float2* sample = nullptr) {
  float fx = __ldg(c.K + 0), cx = __ldg(c.K + 2), fy = __ldg(c.K + 4), cy = __ldg(c.K + 5);
  float x = (px - cx) / fx, y = (py - cy) / fy;
  float dist[4] = {__ldg(c.distortion_params), __ldg(c.distortion_params + 1), __ldg(c.distortion_params + 2),
                   __ldg(c.distortion_params + 3)};
  const float x0 = x, y0 = y;
  if (c.camera_type == 0 || c.camera_type == 1) undistort(x, y, dist);
  // an undistorted pinhole's sample is the pixel position itself
  if (sample) *sample = x == x0 && y == y0 ? make_float2(px, py) : make_float2(fmaf(fx, x, cx), fmaf(fy, y, cy));
  f3 dc;
  if (c.camera_type == 1) {
    float theta = sqrtf(x * x + y * y);
    theta = fminf(3.14159265f, theta);
    float s = (theta < 1e-6f) ? 1.0f : sinf(theta) / theta;
    dc = {x * s, y * s, cosf(theta)};
    if (sample) {
      // the direction is rounded to 2e-7, the sample moves by focal length / cos^2 of the angle for that
      const float qnan = __int_as_float(0x7fc00000);
      const bool exact = dc.z > 0.0f && dc.z * dc.z > 2.5e-5f * fmaxf(fabsf(fx), fabsf(fy));
      *sample = exact ? make_float2(fmaf(fx, dc.x / dc.z, cx), fmaf(fy, dc.y / dc.z, cy)) : make_float2(qnan, qnan);
    }
  } else {
    float l = sqrtf(fmaf(x, x, __fmul_rn(y, y)) + 1.0f);
    dc = {x / l, y / l, 1.0f / l};
  }
  const float* W = c.world_view_transform;
  f3 w = {dot_fma({__ldg(W + 0), __ldg(W + 4), __ldg(W + 8)}, dc), dot_fma({__ldg(W + 1), __ldg(W + 5), __ldg(W + 9)}, dc),
          dot_fma({__ldg(W + 2), __ldg(W + 6), __ldg(W + 10)}, dc)};
  float l = sqrtf(dot_fma(w, w));
  return {w.x / l, w.y / l, w.z / l};
}

// ----------------------------------------------------------------------------
// Per (pixel, record) evaluation shared by forward and backward
// ----------------------------------------------------------------------------
struct Eval {
  float enter, exit, te;  // distances from the offset origin; te is the entry before the clamp at 0
  float dt, tau, alpha;
  float cr, cg, cb;           // colour contribution
};

// The entering and exit distances are plain max/min chains over the four planes:
// a plane the ray crosses inwards (den < 0) bounds the entry, one it crosses outwards
// (den > 0) the exit.  The reference ignores a plane with |den| < 1e-10 unless the
// origin lies outside it, which is a miss (slang/intersect.slang:478-607).  The chains
// give the same answers without the special case: such a plane's distance -D/den is
// huge, positive when the origin is outside (the entry passes the exit: a miss) and
// negative when it is inside (no effect on the maximum), and symmetrically for the
// exit.  A denominator of exactly zero gives +-inf with the sign that rejects the ray
// when the origin is outside and changes nothing when it is inside, provided -0 counts
// as "crossing inwards": the direction of a plane is therefore read from the sign bit
// of den, not from den < 0.  0/0 is NaN, which fmaxf/fminf drop (the reference ignores
// that plane too).
// The four denominators are formed two planes at a time with packed multiply-adds, which round as the
// scalar ones do.
struct Ray {
  float2 x, y, z;  // direction, every component twice
};
__device__ __forceinline__ Ray make_ray(f3 d) { return {{d.x, d.x}, {d.y, d.y}, {d.z, d.z}}; }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
  float2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;"
      : "=l"(reinterpret_cast<unsigned long long&>(r))
      : "l"(reinterpret_cast<unsigned long long&>(a)), "l"(reinterpret_cast<unsigned long long&>(b)),
        "l"(reinterpret_cast<unsigned long long&>(c)));
  return r;
}
__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
  float2 r;
  asm("mul.rn.f32x2 %0, %1, %2;"
      : "=l"(reinterpret_cast<unsigned long long&>(r))
      : "l"(reinterpret_cast<unsigned long long&>(a)), "l"(reinterpret_cast<unsigned long long&>(b)));
  return r;
}
// The hardware's approximations with denormals flushed.  The plain forms (__fdividef, __expf) rescale around denormal
// operands, three to four instructions each time; here a denominator below 1e-38 only occurs as an exact zero, and
// exponentials below 1e-38 are weights that nothing sees.
__device__ __forceinline__ float fast_exp(float x) {
  float r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x * 1.4426950408889634f));
  return r;
}

// 1 / denominator and distance u = -D / denominator from the camera position of the four planes, and the two
// chains: where the ray has entered (ue) and where it leaves (ux).
struct PlaneHits {
  float r[4], u[4];
  bool ent[4];
  float ue, ux;
};
__device__ __forceinline__ PlaneHits plane_hits(const float4 (&rec)[4], const Ray& d) {
  PlaneHits h;
#pragma unroll
  for (int i = 0; i < 4; i += 2) {
    const float4 a = rec[i], b = rec[i + 1];  // (n.x, n.x, n.y, n.y) and (n.z, n.z, -D, -D) of two planes
    const float2 den = fma2({b.x, b.y}, d.z, fma2({a.x, a.y}, d.x, mul2({a.z, a.w}, d.y)));
    h.r[i] = fast_rcp(den.x);
    h.r[i + 1] = fast_rcp(den.y);
    const float2 u = mul2({b.z, b.w}, {h.r[i], h.r[i + 1]});
    h.u[i] = u.x;
    h.u[i + 1] = u.y;
    h.ent[i] = __float_as_int(den.x) < 0;  // sign bit: -0 bounds the entry, +0 the exit
    h.ent[i + 1] = __float_as_int(den.y) < 0;
  }
  h.ue = -1e30f;
  h.ux = 1e30f;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    if (h.ent[i]) h.ue = fmaxf(h.ue, h.u[i]);
    else h.ux = fminf(h.ux, h.u[i]);
  }
  return h;
}

// Distances are first taken from the camera position and shifted by min_t afterwards:
// t = -(D + min_t*den)/den = u - min_t.  A ray that enters the tet after it leaves, or leaves it behind its origin,
// has exit - enter < 0 or = 0, so the sign of the optical depth alone tells a hit; a hit leaves at tx, without a clamp.
// The shift stays: ux - max(ue, min_t) saves the walks an addition per hit (2M tets: forward 2 %, backward 1 %), but rounds
// the length of up to a tenth of the segments otherwise, and with it the optical depth at which a ray ends.
// Returns whether the ray crosses the tet with a positive optical depth.
__device__ __forceinline__ bool slab_test(const float4 (&rec)[4], const Ray& d, float min_t, float density, Eval& e) {
  const PlaneHits h = plane_hits(rec, d);
  e.te = h.ue - min_t;
  e.enter = fmaxf(e.te, 0.0f);
  e.exit = h.ux - min_t;
  e.dt = e.exit - e.enter;
  e.tau = __fmul_rn(density, e.dt);  // never fused into the sum of optical depths
  return e.tau > 0.0f;
}

// For the backward passes: the distances with the reciprocal denominators of the planes that produced them, and
// those planes as one bit each, entering 1 << 2 i, leaving 2 << 2 i (the first plane, in index order, whose
// distance equals the chain's result; where no plane bounds one end it is never differentiated).
struct Crossing {
  float ue, ux, r_e, r_x;
  unsigned faces;
};
__device__ __forceinline__ Crossing slab_planes(const float4 (&rec)[4], const Ray& d) {
  const PlaneHits h = plane_hits(rec, d);
  Crossing c;
  c.ue = h.ue;
  c.ux = h.ux;
  unsigned fe = 64u, fx = 128u;
  c.r_e = c.r_x = h.r[3];
#pragma unroll
  for (int i = 2; i >= 0; --i) {
    const bool in = h.ent[i] && h.u[i] == c.ue, out = !h.ent[i] && h.u[i] == c.ux;
    c.r_e = in ? h.r[i] : c.r_e;
    fe = in ? 1u << (2 * i) : fe;
    c.r_x = out ? h.r[i] : c.r_x;
    fx = out ? 2u << (2 * i) : fx;
  }
  c.faces = fe | fx;
  return c;
}

// Weights of the closed-form segment integral for optical depth x > 0:
//   alpha = exp(-x), phi = (1 - alpha)/x, w0 = phi - alpha, w1 = 1 - phi, and slope = w0/x = -d phi/dx.
// Below x = 0.25 the differences cancel: w1 = x p(x) comes from its Taylor series (truncation < 1e-7 relative) and
// w0 from w0 + w1 = 1 - alpha = x phi = x - x w1, a difference that halves the leading term only; above, both come from the
// fast exponential, each by a multiply-add of its own: w0 falls as 1/x, and as a difference of the sum and w1, two numbers
// near 1, it would lose all precision to an optical depth of 1e7.
__device__ __forceinline__ void segment_weights(float x, float& alpha, float& w0, float& w1, float& slope) {
  alpha = fast_exp(-x);
  // p = 1/2 - x/6 + x^2/24 - x^3/120 + x^4/720 - x^5/5040
  const float p = fmaf(x, fmaf(x, fmaf(x, fmaf(x, fmaf(x, -1.0f / 5040.0f, 1.0f / 720.0f), -1.0f / 120.0f), 1.0f / 24.0f),
                               -1.0f / 6.0f), 0.5f);
  const float inv = fast_rcp(x), rest = 1.0f - alpha, series = __fmul_rn(x, p);
  // both forms are evaluated: the lanes of a warp nearly always need both, and selects cost less than the branch
  const bool thin = x < 0.25f;
  w1 = thin ? series : fmaf(-rest, inv, 1.0f);
  w0 = thin ? fmaf(-x, series, x) - series : fmaf(rest, inv, -alpha);
  slope = thin ? (1.0f - w1) - p : w0 * inv;
}

// Colour of the segment of a hit.  Here and in what it calls the contraction is spelled out, so that every walk that the
// compiler builds from it has the same bits.
__device__ __forceinline__ void integrate(float4 cg, float4 cb, f3 d, float min_t, Eval& e) {
  const float gd = dot_fma({cg.x, cg.y, cg.z}, d);
  const float oe = fmaf(e.enter + min_t, gd, cg.w), ox = fmaf(e.exit + min_t, gd, cg.w);
  float w0, w1, slope;
  segment_weights(e.tau, e.alpha, w0, w1, slope);
  // w0 (base + ox) + w1 (base + oe), channel by channel: the gradient is the same on all of them
  const float w = w0 + w1, o = fmaf(w0, ox, w1 * oe);
  e.cr = fmaf(w, cb.x, o);
  e.cg = fmaf(w, cb.y, o);
  e.cb = fmaf(w, cb.z, o);
}

// The copies write shared memory behind the compiler's back: without the clobbers it may read the destination before the wait,
// or still after the copy that refills it.
__device__ __forceinline__ void cp_async16_l1(void* smem, const void* gmem) {
  uint32_t s = (uint32_t)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
  uint32_t s = (uint32_t)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async4(void* smem, const void* gmem) {
  uint32_t s = (uint32_t)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

constexpr int kWarpsPerBlock = 4;

// 16 pixels of a tile: a block of 4 x 4 where tiles divide into such blocks, else 16 in the order of the tile's rows.  A block
// is touched by fewer tets than a strip, and more of its pixels by each (600k tets, 800 x 800, constant colour, 16 x 16
// tiles: 658 -> 549 us with blocks in place of strips of 16 x 1).
struct Unit {
  int tile;       // linear tile index
  int x, y;       // pixel
  bool inside;    // pixel exists
  int start, len; // tile list
  int sub, subs;  // which 16-pixel group of the tile this half-warp owns, out of how many
};

// The t-th tile to be walked: rows in pairs, tiles of a pair in blocks of 2 x 2, so that the warps of a block have a patch of
// tiles and not a strip, with fewer tets on its border (6.7M tets, 1080p, forward 1.64 -> 1.60 ms, backward 1.80 -> 1.77; 36M,
// 2160p, 6.72 -> 6.62; 21M backward 2.92 -> 2.88; the others the same.  Patches of 4 x 2, 4 x 4 and 8 x 4 give less).
__device__ __forceinline__ int walked_tile(const RmCamera& c, int64_t t) {
  const unsigned width = c.grid_width, rows = c.tile_row_end - c.tile_row_begin;
  const unsigned pair = (unsigned)t / (2 * width), r = (unsigned)t - pair * 2 * width, even = width & ~1u;
  unsigned x = r, y = 2 * pair;
  if (y + 1 < rows) {
    const bool block = r < 2 * even;
    x = block ? 2 * (r >> 2) + (r & 1u) : width - 1;
    y += block ? (r >> 1) & 1u : r - 2 * even;
  }
  return (int)((c.tile_row_begin + y) * width + x);
}

__device__ __forceinline__ Unit make_unit(const RmCamera& c, const int2* __restrict__ ranges, int64_t unit,
                                          int64_t n_units, int subs, int lane16) {
  Unit u;
  u.inside = false;
  u.start = 0;
  u.len = 0;
  u.tile = 0;
  u.x = u.y = 0;
  u.sub = 0;
  u.subs = subs;
  if (unit >= n_units) return u;
  int64_t t = unit / subs;
  int sub = (int)(unit - t * subs);
  u.tile = walked_tile(c, t);
  int ty = u.tile / c.grid_width, tx = u.tile - ty * c.grid_width;
  u.sub = sub;
  int lx, ly;
  if (((c.tile_width | c.tile_height) & 3) == 0) {
    const int across = c.tile_width >> 2, by = sub / across;
    lx = 4 * (sub - by * across) + (lane16 & 3);
    ly = 4 * by + (lane16 >> 2);
  } else {
    const int p = sub * 16 + lane16;
    ly = p / c.tile_width;
    lx = p - ly * c.tile_width;
  }
  u.x = tx * c.tile_width + lx;
  u.y = ty * c.tile_height + ly;
  u.inside = ly < c.tile_height && u.x < c.image_width && u.y < c.image_height;
  int2 rg = __ldg(ranges + u.tile);
  u.start = rg.x;
  u.len = rg.y - rg.x;
  if (u.len > 0 && !(RM_INDEX_OK(rg.x, RM_X_LIST, 0) && RM_INDEX_OK(rg.y - 1, RM_X_LIST, 0))) u.len = 0;
  return u;
}

__device__ __forceinline__ SampleBox halfwarp_sample_box(bool inside, float2 s, float margin) {
  const bool known = inside && s.x == s.x;
  const unsigned lost = __ballot_sync(0xffffffffu, inside && !known) >> (threadIdx.x & 16);
  float x0 = known ? s.x : 3.0e38f, x1 = known ? s.x : -3.0e38f;
  float y0 = known ? s.y : 3.0e38f, y1 = known ? s.y : -3.0e38f;
#pragma unroll
  for (int o = 8; o >= 1; o >>= 1) {
    x0 = fminf(x0, __shfl_xor_sync(0xffffffffu, x0, o));
    x1 = fmaxf(x1, __shfl_xor_sync(0xffffffffu, x1, o));
    y0 = fminf(y0, __shfl_xor_sync(0xffffffffu, y0, o));
    y1 = fmaxf(y1, __shfl_xor_sync(0xffffffffu, y1, o));
  }
  if (lost & 0xFFFFu) return {{0.f, 0.f, 0.f, 0.f}, 3.0e38f};  // only a tet that no ray can hit misses it
  return {{0.5f * (x0 + x1), 0.5f * (y0 + y1), 0.5f * (x1 - x0), 0.5f * (y1 - y0)}, margin};
}

// ----------------------------------------------------------------------------
// Forward
// ----------------------------------------------------------------------------
// A half-warp owns 16 pixels of one tile and walks the tile's list in three stages that
// are decoupled by two small queues in shared memory (ring buffers of 32 slots):
//   1. examination, 16 entries at a time: every lane tests the hull lines of one entry
//      (32 bytes, on their way to shared memory two steps ahead, their tet ids as many
//      before that) against the bounding box of the half-warp's samples (k_pack_records marks
//      the lines of a tet of zero density); survivors go to queue A in list order with their
//      position and their lines;
//   2. when both half-warps hold 16 entries in queue A (or have nothing left to examine),
//      every lane takes one of them and tests the hull lines against each of the 16 sample
//      positions, which gives the mask of the pixels whose ray can touch the tet; entries
//      with an empty mask are dropped, the others go to queue B with their mask;
//   3. when both half-warps hold 16 entries in queue B (or have run dry), the batch staged one
//      round earlier is evaluated and the records of the next (96 bytes each) are staged
//      behind it with 128-bit cp.async copies, which land while stages 1 and 2 of the next
//      round run.  Evaluation: the masks are transposed so that every lane (= pixel) holds
//      the bit set of the batch entries that cover it, and every lane walks its own bits in
//      list order.  Lanes therefore work on different entries at the same time and no lane
//      runs a slab test for a tet that cannot cover its pixel.  A pixel stops at its
//      termination threshold; a half-warp stops examining once all of its pixels have
//      stopped.
// For the backward pass every evaluated batch is appended to the half-warp's hit list:
// the tet ids of the batch and, per pixel, the bit set of the batch entries it hit.
constexpr int kBatch = 16;       // entries staged and evaluated per half-warp and round
constexpr int kRing = 32;        // slots of each candidate queue
// Examination steps whose hull lines are on their way; tet ids are read as many steps before that.  A step is 100 instructions and
// waited 1,360 cycles for its ids and lines, as did stage 2 for its lines, when lines and ids were fetched a step later each and
// stage 2 read its lines from L1: 2M tets, 822 x 1237, 2.01 ms, 6.7M, 1080p, 1.83, 36M, 2160p, 7.39, constant colour, 600k,
// 800 x 800, 0.54; then 1.80, 1.65, 6.72, 0.52, of which the order of a step (copies before the test) is 2 % (1.59 and 6.50 with
// tiles in blocks and lines past L1, below).  Before, 59 % of the issue slots; now 70 %, with 3 % more instructions.  Three steps instead of two are no faster on large grids and leave less of
// L1 (600k, 800 x 800: 377 us with two, 385 with three) and two warps less of the statistics (2M: 2.35 ms and 2.47).
constexpr int kAhead = 2;

// An examination step on its way: hull lines of its entries, first and second 16 bytes apart by a distance at which two lanes
// that copy the two of one entry meet no bank twice, and tet ids, of this step and of the one kAhead later in turn.
struct ExamStep {
  float4 low[32], gap[4], high[32];
  int ids[2][32];
};
// What a warp keeps in shared memory.  What the evaluation loop does not need - hull lines on their way to the
// examination, sample box, hit-list positions - lives here and not in registers.  10 KB: five blocks of four warps per SM.
template <int STRIDE, bool POSITIONS>
struct WalkShared {
  float4 stage[2 * kBatch * STRIDE];
  ExamStep steps[kAhead];                  // [step % kAhead]; the gap of the first two: what `box` and `hits` return
  float4 a_low[2 * kRing], a_high[2 * kRing];  // hull lines of the entries in queue A
  float4 samples[8][2];                    // [pair][half]: two samples each: x0, x1, y0, y1
  uint16_t batch_mask[2 * kBatch];         // entries e and e + 8 of 16 in one word
  int a_id[2 * kRing], b_id[2 * kRing], batch_id[2 * kBatch];
  uint16_t b_mask[2 * kRing];
  int a_pos[POSITIONS ? 2 * kRing : 1], b_pos[POSITIONS ? 2 * kRing : 1], batch_pos[POSITIONS ? 2 * kBatch : 1];

  static_assert(kAhead >= 2, "`hits` are in the gap of the second step");
  __device__ __forceinline__ float4* box(int half) { return &steps[0].gap[2 * half]; }  // centre and half extents, then the margin
  __device__ __forceinline__ int64_t* hits(int half) {  // first id slot and first mask slot of the hit list
    return reinterpret_cast<int64_t*>(&steps[1].gap[half]);
  }
};

// The Tukey power ladder of the constant-colour variant (slang/alphablend_shader.slang:26-33):
// sign(x) |p-1|/p ((|x|/|p-1| + 1)^p - 1).
__device__ __forceinline__ float tukey_power_ladder(float x, float p) {
  const float q = fmaxf(fabsf(p - 1.0f), 1.0754944e-20f);
  const float y = fabsf(p - 1.0f) / p * (__powf(fabsf(x) / q + 1.0f, p) - 1.0f);
  return x > 0.0f ? y : (x < 0.0f ? -y : 0.0f);
}

// Mask of the 16 samples, in pairs (x0, x1, y0, y1), that lie inside (or within the margin of) the convex hull given by
// four lines; NaN lines (cull disabled for the tet) and samples that are not known give set bits.  Two samples per packed
// multiply-add; the sign bits of the four line values together are shifted into the mask (a NaN's is clear).
__device__ __forceinline__ uint32_t hull_sample_mask(float4 l0, float4 l1, const float4 (*__restrict__ samples)[2], int half,
                                                     float margin) {
  HullLines h = unpack_lines(l0, l1);
#pragma unroll
  for (int k = 0; k < 4; ++k) h.c[k] += margin;
  uint32_t outside = 0;
#pragma unroll
  for (int i = 7; i >= 0; --i) {
    const float4 s = samples[i][half];
    float2 v[4];
#pragma unroll
    for (int k = 0; k < 4; ++k)
      v[k] = fma2({h.a[k], h.a[k]}, {s.x, s.y}, fma2({h.b[k], h.b[k]}, {s.z, s.w}, {h.c[k], h.c[k]}));
    auto any = [](float a, float b, float c, float d) {
      return __float_as_uint(a) | __float_as_uint(b) | __float_as_uint(c) | __float_as_uint(d);
    };
    outside = __funnelshift_l(any(v[0].y, v[1].y, v[2].y, v[3].y), outside, 1);
    outside = __funnelshift_l(any(v[0].x, v[1].x, v[2].x, v[3].x), outside, 1);
  }
  return ~outside & 0xFFFFu;
}

// Bit j of the result = bit `lane16` of the mask of entry j of 16; word i (of 8, 16-byte aligned) holds entries i and i + 8.
__device__ __forceinline__ uint32_t transpose_masks(const uint16_t* __restrict__ masks, int lane16) {
  uint32_t bits = 0;
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    const uint4 w = reinterpret_cast<const uint4*>(masks)[q];
    bits |= ((w.x >> lane16) & 0x10001u) << (4 * q);
    bits |= ((w.y >> lane16) & 0x10001u) << (4 * q + 1);
    bits |= ((w.z >> lane16) & 0x10001u) << (4 * q + 2);
    bits |= ((w.w >> lane16) & 0x10001u) << (4 * q + 3);
  }
  return (bits & 0xFFu) | (bits >> 8);
}

// MODE kColor: the interpolated-colour renderer (slang/alphablend_shader_interp.slang).
// MODE kConstColor: the constant-colour debug renderer (slang/alphablend_shader.slang:100-182,
// utils.slang:160-186): records packed with a zero colour gradient, samples at the pixel centres
// (jitter == nullptr), pixel state (rgb, transmittance) with alpha = 1 - exp(-density * dt), four
// distortion moments weighted by transmittance * alpha with the power ladder of the entry distance,
// termination when the transmittance falls below 1/255; out_img = (r, g, b, transmittance) and
// dist_img has four channels.
// MODE kStats: densification statistics (slang/alphablend_shader_interp.slang:433-599,
// internal/render_err.py:119-150): the same walk from the pixel centres with the pixel state starting at
// log-transmittance 1, as the reference has it; every hit adds T = exp(logT_before) * optical_depth times
// (1, err, err^2, -, -, ssim, entry point, exit point, 1, mid point) to row g of tet_err[T,16] and updates
// tet_count[T,2] (hit count, max of int(65535*T)).  The reference issues 14 float and 2 integer atomics per
// (pixel, tet) hit.  Here a hit leaves three scalars, T and T times its two distances, in shared memory; a lane
// per (entry, half row) then adds them up over the 16 pixels, multiplied by constants of the pixel, and issues
// one or three 128-bit reductions.  2M tets, 822 x 1237, a lens: 3.62 ms for a walk of its own over the entries in
// lock-step with 16 sums by shuffles, 2.60 ms for sums pixel by pixel with what was not hit masked out, 2.51 ms for sums of
// two pixels in a packed addition, a slot of zeros in the place of what was not hit.  Then
// a lane per (entry, half row) that adds up all 16 pixels with selections took 2.35 ms, with predicates on the multiply-adds 2.30.
enum ForwardMode { kColor, kConstColor, kStats };
constexpr int kStatsBatch = 8;  // entries whose hits are in shared memory at a time

// float4 per staged record: 6 used, of the statistics, which need no colours, 5; the odd stride spreads the records over the banks
template <ForwardMode MODE>
constexpr int kStageStride = MODE == kStats ? 5 : 7;
using FwdShared = WalkShared<kStageStride<kColor>, true>;
// What a hit leaves, at [pixel] of its entry's row: for part 0 of the sums T twice, for part 1 T times its two distances.  The odd
// stride in units of 16 bytes spreads the entries over the banks.
struct StatsRow {
  float4 hit[16], unused;
};
struct StatsShared : WalkShared<kStageStride<kStats>, false> {  // 13.8 KB; nobody asks for the number of entries walked
  StatsRow rows[2 * kStatsBatch];
  float4 pixel[16][2][2];  // [pixel][half][part]: err, err^2, ssim, 1; ray direction, its x again
};
struct StatsArgs {
  const float *pixel_err, *ssim_err;
  float* tet_err;
  int32_t* tet_count;
};
// How the units of 16 pixels are dealt to warps; the rule is at rm_launch_forward.
//   halves:     two units per warp, one per half: every lane walks its pixel's entries one by one.
//   pairs:      one unit per warp, and two lanes per pixel: each evaluates every other entry that covers the pixel, and
//               what the second has found goes to the first by shuffles, which takes the two through the pixel's state in
//               list order.  Steps and batches of 32 entries in place of 16.  Half the serial chain per
//               unit, which is what a grid that fills the chip once or a few times waits for, for 12 % more issue and
//               shared-memory work per hit (128 x 128 pixels, 13k tets: 54 -> 37 us; 720 x 720 fisheye, 1M tets:
//               414 -> 291 us; 822 x 1237, 2M tets, evenly long lists: 1.87 -> 2.08 ms;
//               constant colour, 600k tets, 800 px, 16 x 16 tiles: 809 -> 654 us).
//   long first: tiles with long lists first, by pairs, the rest by halves.  A unit of 3,000 candidates among units of 100
//               otherwise starts when its turn in the raster comes, and the chip waits for it at the end (6M tets, 1080p:
//               1.88 -> 1.64 ms; 18M: 3.27 -> 2.49 ms).
// A pixel's hits are taken in the same order with the same operations in all of them: which one a call uses cannot be told
// from the bits of its image, so that a frame in bands, each dealt by its own size, is the frame.
// A pixel's state behind a hit: transmittance and distortion moments (dy without a factor of two, dv without one of a third).
// m2: twice the first moment of the density over the segment; of the constant-colour variant the laddered distance.
template <ForwardMode MODE>
__device__ __forceinline__ void update_state(float tau, float alpha, float dens, float m2, float& T, float& logT, float& dx,
                                             float& dy, float& dz, float& dw, float& dv) {
  if (MODE == kConstColor) {
    const float weight = __fmul_rn(T, 1.0f - alpha);
    dx = fmaf(2.0f * weight * m2, dz, dx);
    dy = fmaf(weight, dw, dy);
    dz += weight;
    dw = fmaf(weight, m2, dw);
  } else {
    logT -= tau;
    dx = fmaf(m2, dz, dx);
    dy = fmaf(dens, dw, dy);
    dz += dens;
    dw = fmaf(m2, 0.5f, dw);
    dv = fmaf(dens, tau, dv);
  }
  T *= alpha;
}

template <ForwardMode MODE>
using ForwardShared = typename std::conditional<MODE == kStats, StatsShared, FwdShared>::type;

// The walk of one unit (PAIR), or of the two units of a warp's halves.  Lists longer than `skip_length` are left to others.
// PAST_L1: hull lines are copied past L1; the rule is at lines_past_l1.
template <ForwardMode MODE, bool PAIR, bool PAST_L1>
__device__ __forceinline__ void walk_unit(
    ForwardShared<MODE>& sm, int64_t unit, int skip_length, const int32_t* __restrict__ list,
    const int2* __restrict__ ranges, const float4* __restrict__ records, const RmCamera& rcam,
    const float2* __restrict__ jitter, float4* __restrict__ out_img, float* __restrict__ dist_img,
    int32_t* __restrict__ n_contrib, int32_t* __restrict__ hit_counts, int32_t* __restrict__ hit_ids,
    uint16_t* __restrict__ hit_masks, uint8_t* __restrict__ tet_flags, int subs, int64_t n_units, float pre_multi,
    float ladder_p, const StatsArgs& stats) {
  constexpr unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  constexpr int kEntries = PAIR ? 32 : kBatch;     // entries per step, one per lane of the unit
  constexpr int kSlots = PAIR ? 2 * kRing : kRing;  // of each queue of the unit
  const int half = PAIR ? 0 : lane >> 4, lane16 = lane & 15;  // unit of the warp, pixel of the unit
  const int el = lane & (kEntries - 1);
  const bool second = PAIR && lane >= 16;  // the lane that takes the later entry of two
  const unsigned below = (1u << el) - 1u;
  auto unit_ballot = [&](bool p) {
    const unsigned b = __ballot_sync(FULL, p);
    return PAIR ? b : (b >> (16 * half)) & 0xFFFFu;
  };
  int *const a_id = sm.a_id + half * kRing, *const a_pos = sm.a_pos + half * kRing;
  int *const b_id = sm.b_id + half * kRing, *const b_pos = sm.b_pos + half * kRing;
  float4 *const a_low = sm.a_low + half * kRing, *const a_high = sm.a_high + half * kRing;
  uint16_t* const b_mask = sm.b_mask + half * kRing;
  int *const batch_id = sm.batch_id + half * kBatch, *const batch_pos = sm.batch_pos + half * kBatch;
  uint16_t* const batch_mask = sm.batch_mask + half * kBatch;
  constexpr int kStride = kStageStride<MODE>;
  float4* const stage = sm.stage + half * kBatch * kStride;
  Unit u = make_unit(rcam, ranges, unit, n_units, subs, lane16);
  if (u.len > skip_length) {
    u.inside = false;
    unit = n_units;
  }

  f3 d = {0.f, 0.f, 1.f};
  {
    float2 sample = make_float2(0.f, 0.f);
    if (u.inside) {
      float2 j = jitter ? __ldg(jitter + (int64_t)u.y * rcam.image_width + u.x) : make_float2(0.5f, 0.5f);
      d = ray_direction(rcam, (float)u.x + j.x, (float)u.y + j.y, &sample);
    }
    float* sp = reinterpret_cast<float*>(&sm.samples[lane16 >> 1][half]) + (lane16 & 1);
    sp[0] = sample.x;
    sp[2] = sample.y;
    const SampleBox box = halfwarp_sample_box(u.inside, sample, rcam.camera_type == 1 ? kFisheyeMargin : kPixelMargin);
    if (lane16 == 0) {
      sm.box(half)[0] = box.box;
      sm.box(half)[1].x = box.margin;
      // Hit list of this half-warp: the tet ids of every evaluated batch at [first, first + n_ent), and for batch b
      // the 16 per-pixel bit sets behind the mask slot.  Every batch but the last holds 16 entries.
      const int64_t first = (int64_t)u.start * u.subs + (int64_t)u.sub * u.len;
      sm.hits(half)[0] = first;
      sm.hits(half)[1] = first + 16 * ((int64_t)u.tile * u.subs + u.sub);
    }
  }
  const Ray ray = make_ray(d);
  const float min_t = rcam.min_t;

  if constexpr (MODE == kStats) {
    float perr = 0.f, serr = 0.f;
    if (u.inside) {
      const int64_t pix = (int64_t)u.y * rcam.image_width + u.x;
      perr = __ldg(stats.pixel_err + pix);
      serr = __ldg(stats.ssim_err + pix);
    }
    sm.pixel[lane16][half][0] = make_float4(perr, perr * perr, serr, 1.0f);
    sm.pixel[lane16][half][1] = make_float4(d.x, d.y, d.z, d.x);
  }

  float sr = 0.f, sg = 0.f, sb = 0.f, logT = MODE == kStats ? 1.0f : 0.0f, T = MODE == kStats ? 2.718281828f : 1.0f;
  float dx = 0.f, dy = 0.f, dz = 0.f, dw = 0.f, dv = 0.f;
  int contrib = 0;
  bool active = u.inside;
  unsigned act16 = unit_ballot(active) & 0xFFFFu;  // pixels of this half still walking
  bool fetching = act16 != 0;
  int n_ent = 0;  // entries in the hit list

  // Examination: entry src + el is the one this lane examines next.  The hull lines of that step and of the kAhead - 1 behind it
  // are in sm.steps or on their way, and so are the tet ids of the kAhead steps behind those.  All of it by asynchronous copies, two
  // lanes for the lines of an entry, so that a sector is one access.  Behind the end of the list its last entry is copied.
  // A negative id in a caller's list names no tet: the lines of tet 0 are copied for it, and stage 2 drops it (a test per entry
  // that has survived; dropped by the examination it costs 0.8 % of the walk and not 0.4).
  int src = 0;
  int qa_h = 0, qa_n = 0, qb_h = 0, qb_n = 0;  // ring heads and fill levels (the same in all lanes of the half)
  if (!fetching) u.len = 0;
  const int last = u.len - 1;
  const int32_t* const list_at = list + u.start;
  const float4* const lines_at = records + kLinesAt + (el & 1);
  ExamStep* step = sm.steps;
  int turn = 0;  // which of the step's ids are its own
  const int pair_lane = lane - el + (el >> 1);  // entry whose lines this lane copies, and the one kEntries / 2 on
  auto fetch = [&](int first, ExamStep* st, int at) {  // lines of the step at `first` with the ids [at], ids of kAhead steps on
    float4* const to = (el & 1 ? st->high : st->low) + pair_lane;
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const int id = max(st->ids[at][pair_lane + k * (kEntries / 2)], 0);
      if (!RM_INDEX_OK(id, RM_X_TETS, 1)) continue;
      if (PAST_L1) cp_async16(to + k * (kEntries / 2), lines_at + record_at(id));
      else cp_async16_l1(to + k * (kEntries / 2), lines_at + record_at(id));
    }
    cp_async4(&st->ids[at ^ 1][lane], list_at + min(first + kAhead * kEntries + el, last));
  };
  if (u.len > 0) {
#pragma unroll
    for (int k = 0; k < kAhead; ++k) sm.steps[k].ids[0][lane] = __ldg(list_at + min(k * kEntries + el, last));
  }
  __syncwarp();
#pragma unroll
  for (int k = 0; k < kAhead; ++k) {
    if (u.len > 0) fetch(k * kEntries, sm.steps + k, 0);
    cp_async_commit();
  }

  int n_cur = 0;   // entries of the staged batch
  int since = kAhead;   // examination steps since records were staged
  __syncwarp();
  for (;;) {
    {
      const bool done = !fetching || (n_cur == 0 && qb_n == 0 && qa_n == 0 && src >= u.len);
      if (__all_sync(FULL, done)) break;
    }
    // ---- stages 1 and 2: until both halves hold a full batch in queue B or have run dry
    for (;;) {
      const bool hungry = fetching && qb_n < kEntries;
      for (;;) {
        const bool examine = hungry && qa_n < kEntries && src < u.len;
        if (!__any_sync(FULL, examine)) break;
        // Copies are committed by all lanes together.  Those of this step lie behind kAhead - 1 later ones; where records were
        // staged since, their copies count as one of these, and a later step's are waited for, which began long before them.
        cp_async_wait<kAhead - 1>();
        __syncwarp();
        const float4 l0 = step->low[lane], l1 = step->high[lane];
        const int id = step->ids[turn][lane], pos = src + el;
        __syncwarp();  // all lanes have read; the copies, which depend on nothing else, come before the long chain of the test
        if (examine) {
          fetch(src + kAhead * kEntries, step, turn ^ 1);
          src += kEntries;
          if (++step == sm.steps + kAhead) {
            step = sm.steps;
            turn ^= 1;
          }
        }
        cp_async_commit();
        const bool cand = examine && pos <= last && !hull_misses_box(l0, l1, {sm.box(half)[0], sm.box(half)[1].x}) &&
                          RM_INDEX_OK(max(id, 0), RM_X_TETS, 1);
        const unsigned cb = unit_ballot(cand);
        if (cand) {
          const int slot = (qa_h + qa_n + __popc(cb & below)) & (kSlots - 1);
          a_id[slot] = id;
          if (MODE != kStats) a_pos[slot] = pos;
          a_low[slot] = l0;
          a_high[slot] = l1;
        }
        qa_n += __popc(cb);
        ++since;
      }
      const bool need_b = hungry && qa_n > 0;
      if (!__any_sync(FULL, need_b)) break;
      __syncwarp();
      const int take_a = need_b ? min(qa_n, kEntries) : 0;
      uint32_t m = 0;
      int cid = 0, cpos = 0;
      if (el < take_a) {
        const int slot = (qa_h + el) & (kSlots - 1);
        cid = a_id[slot];
        if (MODE != kStats) cpos = a_pos[slot];
        const float margin = rcam.camera_type == 1 ? kFisheyeMargin : kPixelMargin;
        m = hull_sample_mask(a_low[slot], a_high[slot], sm.samples, half, margin) & (cid >= 0 ? act16 : 0u);
      }
      const unsigned lb = unit_ballot(m != 0u);
      if (m) {
        const int slot = (qb_h + qb_n + __popc(lb & below)) & (kSlots - 1);
        b_id[slot] = cid;
        if (MODE != kStats) b_pos[slot] = cpos;
        b_mask[slot] = (uint16_t)m;
      }
      qa_h = (qa_h + take_a) & (kSlots - 1);
      qa_n -= take_a;
      qb_n += __popc(lb);
      __syncwarp();
    }
    // the staged records have landed; up to kAhead later copies of hull lines may still be on their way
    static_assert(kAhead <= 3, "one case for each number of later copies that may leave those of the records on their way");
    if (since == 0) cp_async_wait<0>(); else if (since == 1) cp_async_wait<1>(); else if (since == 2) cp_async_wait<2>();
    __syncwarp();
    // ---- stage 3a: evaluate the batch staged one round ago; every lane walks the entries covering its pixel
    uint32_t bits = (active && n_cur > 0) ? __brev(transpose_masks(batch_mask + (second ? kBatch : 0), lane16)) : 0u;  // entry j: bit 31 - j
    if constexpr (PAIR) {
      const uint32_t other = __shfl_xor_sync(FULL, bits, 16);
      bits = second ? other | (bits >> 16) : bits | (other >> 16);
    }
    uint32_t hitbits = bits;  // nearly every candidate is a hit: the others are taken out
    if constexpr (PAIR) {
      // every other entry of the pixel, from the first or from the second
      uint32_t odd = bits ^ (bits >> 1);
      odd ^= odd >> 2;
      odd ^= odd >> 4;
      odd ^= odd >> 8;
      odd ^= odd >> 16;  // parity of the number of entries up to and with this one
      uint32_t mine = bits & (second ? ~odd : odd), missed = 0;
      while (__any_sync(FULL, mine != 0u)) {
        const int j = __clz(mine);
        Eval e;
        e.tau = e.cr = e.cg = e.cb = 0.f;
        e.alpha = 1.f;  // set by hits alone
        float dens = 0.f, m2 = 0.f;
        if (mine) {
          const uint32_t bit = 0x80000000u >> j;
          mine ^= bit;
          const float4* rec = stage + j * kStride;
          const float4 pl[4] = {rec[0], rec[1], rec[2], rec[3]};
          const float4 cg = rec[4], cb = rec[5];
          if (slab_test(pl, ray, min_t, cb.w, e)) {
            integrate(cg, cb, d, min_t, e);
            dens = cb.w;
            // twice the first moment; of the constant-colour variant the laddered distance
            m2 = MODE == kConstColor ? tukey_power_ladder(e.enter * pre_multi, ladder_p) : dens * (e.exit + e.enter);
          } else {
            e.tau = 0.f;
            missed |= bit;
          }
        }
        // The first lane of a pixel takes its two entries in list order, with the operations of the walk by halves: the bits of
        // an image do not depend on how its units are dealt.  (The second lane goes along; its state is not used.)
        const float o_tau = __shfl_xor_sync(FULL, e.tau, 16), o_alpha = __shfl_xor_sync(FULL, e.alpha, 16);
        const float o_dens = __shfl_xor_sync(FULL, dens, 16), o_m2 = __shfl_xor_sync(FULL, m2, 16);
        const float o_r = __shfl_xor_sync(FULL, e.cr, 16), o_g = __shfl_xor_sync(FULL, e.cg, 16);
        const float o_b = __shfl_xor_sync(FULL, e.cb, 16);
        // An entry that the pixel misses adds zeros, which costs less than a branch (60k tets, 203 x 317: 103 us, with branches
        // 115); it changes nothing as long as no moment has overflowed.
        auto take = [&](float tau, float alpha, float dens, float m2, float r, float g, float b) {
          sr = fmaf(r, T, sr);
          sg = fmaf(g, T, sg);
          sb = fmaf(b, T, sb);
          update_state<MODE>(tau, alpha, dens, m2, T, logT, dx, dy, dz, dw, dv);
          return MODE == kConstColor ? T < 1.0f / 255.0f : logT < -5.5f;
        };
        const bool early = take(e.tau, e.alpha, dens, m2, e.cr, e.cg, e.cb);
        const bool late = take(early ? 0.0f : o_tau, early ? 1.0f : o_alpha, early ? 0.0f : o_dens, early ? 0.0f : o_m2,
                               early ? 0.0f : o_r, early ? 0.0f : o_g, early ? 0.0f : o_b);
        const unsigned ended = __ballot_sync(FULL, active && !second && late);
        if (ended) {
          const int at = __shfl_sync(FULL, (int)early, lane16) ? lane16 : lane16 + 16;
          const int last = __shfl_sync(FULL, j, at);  // the entry at which the pixel has ended
          if ((ended >> lane16) & 1u) {
            active = false;
            contrib = batch_pos[last] + 1;  // entries walked, the terminating one included
            hitbits &= ~(0x7FFFFFFFu >> last);
            mine = 0;
          }
        }
      }
      hitbits &= ~(missed | __shfl_xor_sync(FULL, missed, 16));
      __syncwarp();
    } else
    // kStats: entries 0..7 first, their sums, then 8..15
#pragma unroll 1
    for (int sub = 0; sub < (MODE == kStats ? 2 : 1); ++sub) {
      const uint32_t floor = MODE == kStats && sub == 0 ? 0x00FFFFFFu : 0u;
      while (bits > floor) {
        const int b = 31 - __clz(bits), j = 31 - b;
        bits ^= 1u << b;
        const float4* rec = stage + j * kStride;
        const float4 pl[4] = {rec[0], rec[1], rec[2], rec[3]};
        const float4 cg = rec[4], cb = rec[kStride == 5 ? 4 : 5];
        Eval e;
        if (slab_test(pl, ray, min_t, cb.w, e)) {
          if (MODE == kStats) {
            e.alpha = fast_exp(-e.tau);
          } else {
            integrate(cg, cb, d, min_t, e);
            sr = fmaf(e.cr, T, sr);
            sg = fmaf(e.cg, T, sg);
            sb = fmaf(e.cb, T, sb);
          }
          bool finished;
          if constexpr (MODE == kStats) {
            const float Tw = T * e.tau;
            sm.rows[half * kStatsBatch + (j & 7)].hit[lane16] = make_float4(Tw, Tw, Tw * (e.enter + min_t), Tw * (e.exit + min_t));
            logT -= e.tau;
            T *= e.alpha;
            finished = logT < -5.5f;
          } else {
            const float m2 = MODE == kConstColor ? tukey_power_ladder(e.enter * pre_multi, ladder_p) : cb.w * (e.exit + e.enter);
            update_state<MODE>(e.tau, e.alpha, cb.w, m2, T, logT, dx, dy, dz, dw, dv);
            finished = MODE == kConstColor ? T < 1.0f / 255.0f : logT < -5.5f;
          }
          if (finished) {
            active = false;
            if (MODE != kStats) contrib = batch_pos[j] + 1;  // entries walked, the terminating one included
            hitbits ^= bits;
            bits = 0;
          }
        } else {
          hitbits ^= 1u << b;
        }
      }
      __syncwarp();
      if constexpr (MODE == kStats) {
        // part 0 of an entry sums T, err, err^2 and ssim, part 1 entry and exit points
        const int ent = lane16 >> 1, part = lane16 & 1;
        unsigned mine = 0;
#pragma unroll
        for (int e = 0; e < kStatsBatch; ++e) {
          const unsigned col = __ballot_sync(FULL, (hitbits >> (31 - 8 * sub - e)) & 1u);
          if (ent == e) mine = col;
        }
        mine = (mine >> (16 * half)) & 0xFFFFu;
        // part 0: v = (T, T), x, y, z its sums with err, err^2 and ssim, u without; part 1: v = T times the two distances, x, y, z
        // and u, v, w their sums with the ray direction.  Even and odd pixels apart: two short sums are rounded less than a long one.
        struct Sums { float x, y, z, u, v, w, most; } sums[2];
        sums[0] = sums[1] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        const float2* const row = reinterpret_cast<const float2*>(sm.rows[half * kStatsBatch + ent].hit) + part;
#pragma unroll
        for (int p = 0; p < 16; ++p) {
          const float4 con = sm.pixel[p][half][part];
          const float2 v = row[2 * p];
          Sums& t = sums[p & 1];
          asm("{\n\t.reg .pred p;\n\t.reg .b32 t;\n\t"
              "and.b32 t, %7, %8;\n\tsetp.ne.u32 p, t, 0;\n\t"
              "@p fma.rn.f32 %0, %9, %11, %0;\n\t"
              "@p fma.rn.f32 %1, %9, %12, %1;\n\t"
              "@p fma.rn.f32 %2, %9, %13, %2;\n\t"
              "@p fma.rn.f32 %3, %10, %14, %3;\n\t"
              "@p fma.rn.f32 %4, %10, %12, %4;\n\t"
              "@p fma.rn.f32 %5, %10, %13, %5;\n\t"
              "@p max.f32 %6, %6, %9;\n\t}"
              : "+f"(t.x), "+f"(t.y), "+f"(t.z), "+f"(t.u), "+f"(t.v), "+f"(t.w), "+f"(t.most)
              : "r"(mine), "r"(1u << p), "f"(v.x), "f"(v.y), "f"(con.x), "f"(con.y), "f"(con.z), "f"(con.w));
        }
        const f3 s1 = {sums[0].x + sums[1].x, sums[0].y + sums[1].y, sums[0].z + sums[1].z};
        const f3 s2 = {sums[0].u + sums[1].u, sums[0].v + sums[1].v, sums[0].w + sums[1].w};
        const float most = fmaxf(sums[0].most, sums[1].most), sum = __shfl_sync(FULL, s2.x, lane & ~1);  // part 0's
        const float ssim = __shfl_xor_sync(FULL, s1.z, 1);  // part 0's, needed in a row that part 1 writes
        if (mine) {
          const int64_t id = batch_id[8 * sub + ent];
          float4* row = reinterpret_cast<float4*>(stats.tet_err + 16 * id);
          if (part == 0) {
            atomicAdd(row, make_float4(sum, s1.x, s1.y, 0.0f));
            atomicAdd(stats.tet_count + 2 * id, __popc(mine));
            atomicMax(stats.tet_count + 2 * id + 1, (int)(65535.0f * most));
          } else {
            const f3 cam = {__ldg(rcam.cam_pos), __ldg(rcam.cam_pos + 1), __ldg(rcam.cam_pos + 2)};
            const f3 a = cam * sum + s1, b = cam * sum + s2, m = (a + b) * 0.5f;  // entry, exit and mid points
            atomicAdd(row + 1, make_float4(0.0f, ssim, a.x, a.y));
            atomicAdd(row + 2, make_float4(a.z, b.x, b.y, b.z));
            atomicAdd(row + 3, make_float4(sum, m.x, m.y, m.z));
          }
        }
        __syncwarp();
      }
    }
    if (MODE == kColor && hit_ids && n_cur > 0) {  // append the batch to the hit list
      const int64_t hslot = sm.hits(half)[0] + n_ent + el, mslot = sm.hits(half)[1] + n_ent + el;
      if (el < n_cur && RM_INDEX_OK(hslot, RM_X_HIT_IDS, 2)) {
        const int id = batch_id[el];
        hit_ids[hslot] = id;
        tet_flags[id] = 1;  // this tet's record-gradient row is cleared and read by the backward pass
      }
      if ((!second || n_cur > kBatch) && RM_INDEX_OK(mslot, RM_X_HIT_MASKS, 3))
        hit_masks[mslot] = (uint16_t)(__brev(hitbits) >> (second ? 16 : 0));  // n_ent is a multiple of 16 here
      n_ent += n_cur;
    }
    act16 = unit_ballot(active) & 0xFFFFu;
    fetching = act16 != 0;
    __syncwarp();
    // ---- stage 3b: stage the next batch, the first min(qb_n, 16) entries of queue B; it lands while stages 1 and 2
    // of the next round run
    const int take = fetching ? min(qb_n, kEntries) : 0;
    uint32_t mask = 0;
    if (el < take) {
      const int slot = (qb_h + el) & (kSlots - 1);
      batch_id[el] = b_id[slot];
      if (MODE != kStats) batch_pos[el] = b_pos[slot];
      mask = b_mask[slot];
    }
    batch_mask[(el & 16) + 2 * (el & 7) + ((el >> 3) & 1)] = (uint16_t)mask;
#pragma unroll
    for (int k = 0; k < 2; ++k) {  // two lanes for the record of an entry
      const int e = (el >> 1) + k * (kEntries / 2);
      if (e < take) {
        const float4* src_rec = records + record_at(b_id[(qb_h + e) & (kSlots - 1)]) + (el & 1);
        float4* dst = stage + e * kStride + (el & 1);
        cp_async16(dst, src_rec);
        cp_async16(dst + 2, src_rec + 2);
        if (kStride == 7) cp_async16(dst + 4, src_rec + 4);
        else if (el & 1) cp_async16(dst + 3, src_rec + 4);  // density; the colours are not staged
      }
    }
    cp_async_commit();
    since = 0;
    qb_h = (qb_h + take) & (kSlots - 1);
    qb_n -= take;
    n_cur = take;
  }
  cp_async_wait<0>();
  if (active) contrib = u.len;  // walked the whole list

  if (MODE == kStats) return;
  const int64_t pix = (int64_t)u.y * rcam.image_width + u.x;
  if (hit_counts && el == 0 && unit < n_units && RM_INDEX_OK((int64_t)u.tile * u.subs + u.sub, RM_X_UNITS, 4))
    hit_counts[(int64_t)u.tile * u.subs + u.sub] = n_ent;
  dy *= 2.0f;  // the factors common to all terms of these moments
  dv *= 1.0f / 3.0f;
  if (u.inside && !second) {
    if (MODE == kConstColor) {
      out_img[pix] = make_float4(sr, sg, sb, T);
      reinterpret_cast<float4*>(dist_img)[pix] = make_float4(dx, dy, dz, dw);
    } else {
      out_img[pix] = make_float4(sr, sg, sb, logT);
      float* o = dist_img + 5 * pix;
      o[0] = dx; o[1] = dy; o[2] = dz; o[3] = dw; o[4] = dv;
    }
    n_contrib[pix] = contrib;
  }
}

// Units by halves or by pairs.  A block holds its place until its last warp is done: two warps where units are long and many
// (statistics, 2M tets: 2590 us with four, 2566 with two, 2563 with one), four where neighbouring units that share records
// count (600k tets, 800 x 800, pairs: 416 us with four, 435 with two, 469 with one).
template <ForwardMode MODE>
constexpr int kFwdWarps = MODE == kStats ? 2 : kWarpsPerBlock;
template <ForwardMode MODE, bool PAIR, bool PAST_L1>
__global__ void __launch_bounds__(kFwdWarps<MODE> * 32, (MODE == kStats ? 16 : 20) / kFwdWarps<MODE>)
k_forward(const int32_t* __restrict__ list, const int2* __restrict__ ranges, const float4* __restrict__ records, RmCamera rcam,
          const float2* __restrict__ jitter, float4* __restrict__ out_img, float* __restrict__ dist_img,
          int32_t* __restrict__ n_contrib, int32_t* __restrict__ hit_counts, int32_t* __restrict__ hit_ids,
          uint16_t* __restrict__ hit_masks, uint8_t* __restrict__ tet_flags, int subs, int64_t n_units, float pre_multi,
          float ladder_p, StatsArgs stats) {
  extern __shared__ __align__(16) unsigned char smem_fwd[];
  const int warp = threadIdx.x >> 5, half = (threadIdx.x >> 4) & 1;
  const int64_t at = (int64_t)blockIdx.x * kFwdWarps<MODE> + warp;
  walk_unit<MODE, PAIR, PAST_L1>(reinterpret_cast<ForwardShared<MODE>*>(smem_fwd)[warp], PAIR ? at : 2 * at + half, INT_MAX, list, ranges,
                        records, rcam, jitter, out_img, dist_img, n_contrib, hit_counts, hit_ids, hit_masks, tet_flags, subs,
                        n_units, pre_multi, ladder_p, stats);
}

// Long first: the first `long_blocks` of the grid take the tiles whose list is longer than `long_list`.
// 92 registers, as the walk by halves takes in a kernel of its own.  20 warps fit an SM in blocks of two or of four; with four,
// neighbouring tiles share more (two and four: 2M tets 1805 and 1793 us, 6.7M 1631 and 1616, 21M 2324 and 2287, 36M 6523 and 6485).
constexpr int kLongFirstWarps = 4;
template <bool PAST_L1>
__global__ void __maxnreg__(92)
k_forward_long_first(const int32_t* __restrict__ list, const int2* __restrict__ ranges, const float4* __restrict__ records, RmCamera rcam,
                     const float2* __restrict__ jitter, float4* __restrict__ out_img, float* __restrict__ dist_img,
                     int32_t* __restrict__ n_contrib, int32_t* __restrict__ hit_counts, int32_t* __restrict__ hit_ids,
                     uint16_t* __restrict__ hit_masks, uint8_t* __restrict__ tet_flags, int subs, int64_t n_units, int long_list,
                     int long_blocks) {
  extern __shared__ __align__(16) unsigned char smem_fwd[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  FwdShared& sm = reinterpret_cast<FwdShared*>(smem_fwd)[warp];
  // Warp w of the first blocks looks through units w, w + walkers, ..., 32 at a time: the tiles of a region with long lists
  // go to different warps.
  const int64_t walkers = (int64_t)long_blocks * kLongFirstWarps;
  int64_t at = (int64_t)blockIdx.x * kLongFirstWarps + warp;
  if (at < walkers) {
    for (; at < n_units; at += 32 * walkers) {
      const int64_t u = at + lane * walkers;
      const int2 rg = u < n_units ? __ldg(ranges + walked_tile(rcam, u / subs)) : make_int2(0, 0);
      unsigned found = __ballot_sync(0xffffffffu, rg.y - rg.x > long_list);
      while (found) {
        const int64_t unit = at + (__ffs(found) - 1) * walkers;
        found &= found - 1;
        walk_unit<kColor, true, PAST_L1>(sm, unit, INT_MAX, list, ranges, records, rcam, jitter, out_img, dist_img, n_contrib, hit_counts,
                                hit_ids, hit_masks, tet_flags, subs, n_units, 0.0f, 0.0f, StatsArgs{});
        __syncwarp();
      }
    }
    return;
  }
  at = (int64_t)(blockIdx.x - (unsigned)long_blocks) * kLongFirstWarps + warp;
  walk_unit<kColor, false, PAST_L1>(sm, at * 2 + (lane >> 4), long_list, list, ranges, records, rcam, jitter, out_img, dist_img, n_contrib,
                           hit_counts, hit_ids, hit_masks, tet_flags, subs, n_units, 0.0f, 0.0f, StatsArgs{});
}

// ----------------------------------------------------------------------------
// Backward
// ----------------------------------------------------------------------------
// A half-warp walks the hit list of its 16 pixels from the last entry to the first, eight entries at a time, in
// two phases that divide the work differently:
//   A. lane = pixel.  Every lane walks its own bits of the eight entries, last first: slab test and segment
//      integral again, state undone, the chain rule down to the scalars that multiply constants of the pixel.
//      With the ray direction d and the upstream colour gradient g of the pixel, a hit contributes
//        to its entering and its leaving plane   (uq d, q)     with q = -dL/dt / den, u = distance from the camera
//        to the colour gradient and its offset   (a d, w G)    with G = g.r + g.g + g.b
//        to the base colour and the density      (w g, b)
//      so seven floats leave for shared memory, and the two plane numbers as one byte.
//   B. lane = (entry, half of its row).  The lane adds up its half of the entry's 24 record gradients over the 16
//      pixels, in registers, reading each hit's scalars and the pixel's constants, and adds the sums to the row
//      in global memory with 128-bit reductions: one per plane that the entry has hits on, two for the colours.
// Lanes of phase A are on different entries at the same time, so none waits for entries that its pixel missed, and
// phase B needs no shuffles and no test of which pixels share faces.  Issue slots bound the kernel, so what phase B does per
// pixel is cut to loads, tests and additions:
//   * A ray in front of the near plane enters through planes that face the camera and leaves through the others, which the
//     sign of a plane's D tells.  A lane therefore loads the pair of its plane (8 bytes) and no other, and one bit of the
//     pixel's byte says whether it counts: a predicate on the multiply-adds, where a selection between both pairs and zero
//     takes eight instructions a pixel.
// A near plane behind the camera (BEHIND) has rays that enter and leave on the same side of it: the few entries with such hits
// get a second sum over the other pairs, behind the first (2M tets, min_t = -0.25: 2.33 ms; a second sum for every entry 2.99; 60k
// 101 and 123 us; the second sum in the first one's registers, which do not hold it, 2.87 ms).
// (u = -D / den, so q u = dL/dt u^2 / D, and without the reciprocals, whose pick by plane costs six instructions a hit, 2M tets
// would take 2.33 ms; but the sums, divided by D at the end, are 3 % further from 64 bits.)
// With selections in phase B and 8 ballots a round for who has hit what: 2M tets, 822 x 1237,
// 2.70 ms, 6.7M, 1080p, 2.14, 21M 3.61, a medium scene 1.04e9 warp instructions; then 2.43, 1.92, 3.07 ms, 0.9e9; 2.28, 1.77,
// 2.88 and 0.87e9 with fewer instructions per hit, the hit list's loads first, tiles in blocks.  (A lock-step walk over the entries
// with a reduction per step took twice that.)
constexpr int kBwdBatch = 8;          // entries per half-warp and round
constexpr int kBwdStageStride = 7;    // float4 per staged record (6 used), as in the forward kernel

// What phase A leaves of an entry: [pixel] (uq, q) of the entering and of the leaving plane, and (a, b, w, w).  The odd stride
// in units of 16 bytes spreads the entries over the banks.
struct BwdRow {
  float4 planes[16], fields[16], unused;
};
struct BwdShared {                              // 11 KB: five blocks of four warps per SM, 19 of one warp (a block takes 1 KB more)
  float4 stage[2 * kBwdBatch * kBwdStageStride];  // refilled while phase B runs; behind an entry's record, its 16 face bytes
  BwdRow rows[2 * kBwdBatch];
  float4 pixel[16][2][2];                         // [pixel][half][0: d, 1; 1: g, G]
};
constexpr int kFacesAt = 6;  // of an entry's staged record, in float4: a byte per pixel, entering plane 1 << 2 i, leaving 2 << 2 i

// s + v (x, y, z1) where the word has one of the bits, v.x for the first three components and v.y for the last, whose constant
// of the pixel is z1.y.
__device__ __forceinline__ void add_where(unsigned word, unsigned bits, float2 v, float x, float y, float2 z1, float& sx, float& sy,
                                          float2& sz) {
  asm("{\n\t.reg .pred p;\n\t.reg .b32 t;\n\t"
      "and.b32 t, %3, %4;\n\tsetp.ne.u32 p, t, 0;\n\t"
      "@p fma.rn.f32 %0, %5, %6, %0;\n\t"
      "@p fma.rn.f32 %1, %5, %7, %1;\n\t"
      "@p fma.rn.f32x2 %2, %8, %9, %2;\n\t}"
      : "+f"(sx), "+f"(sy), "+l"(reinterpret_cast<unsigned long long&>(sz))
      : "r"(word), "r"(bits), "f"(v.x), "f"(x), "f"(y), "l"(reinterpret_cast<unsigned long long&>(v)),
        "l"(reinterpret_cast<unsigned long long&>(z1)));
}
// PAIR: one unit per warp, 16 entries a round and two lanes per pixel, each on every other entry of the pixel, the last
// first; what the two entries change of the state is handed over by shuffles.  Both phases then take half as many rounds in
// a row (13k tets, 128 x 128: 70 -> 49 us; 60k, 203 x 317: 154 -> 123 us; 2M, 300 x 300: 543 -> 459 us).
// On its small grids a block of one warp: units of uneven length then do not hold each other's places (with selections in phase B,
// 13k tets, 128 x 128: 49.3 us with four, 45.4 with one; 2M of a scene, 300 x 300: 451 and 445, 430 x 430: 717 and 715; 60k, 203 x 317: the same).
// Large grids lose by it what neighbouring units share (6M: 2202 us with four, 2245 with one).
template <bool PAIR>
constexpr int kBwdWarps = PAIR ? 1 : kWarpsPerBlock;
template <bool PAIR, bool BEHIND>
__global__ void __launch_bounds__(kBwdWarps<PAIR> * 32, PAIR ? 19 : 5)
k_backward(const int2* __restrict__ ranges, const float4* __restrict__ records, RmCamera rcam,
           const float2* __restrict__ jitter, const float4* __restrict__ out_img, const float* __restrict__ dist_img,
           const int32_t* __restrict__ hit_counts, const int32_t* __restrict__ hit_ids,
           const uint16_t* __restrict__ hit_masks, const float4* __restrict__ g_img, const float* __restrict__ g_dist,
           float* __restrict__ grec, int subs, int64_t n_units) {
  after_previous();
  extern __shared__ __align__(16) unsigned char smem_bwd[];
  constexpr unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  constexpr int kEntries = PAIR ? 2 * kBwdBatch : kBwdBatch;
  const int half = PAIR ? 0 : lane >> 4, lane16 = lane & 15;  // unit of the warp, pixel of the unit
  const bool second = PAIR && lane >= 16;
  BwdShared& sm = reinterpret_cast<BwdShared*>(smem_bwd)[warp];
  float4* const staged = sm.stage + half * kBwdBatch * kBwdStageStride;
  BwdRow* const rows = sm.rows + half * kBwdBatch;
  const int64_t unit = ((int64_t)blockIdx.x * kBwdWarps<PAIR> + warp) * (PAIR ? 1 : 2) + half;
  Unit u = make_unit(rcam, ranges, unit, n_units, subs, lane16);

  // The half-warp's hit list (written by the forward pass: the batches of 16 it evaluated, each with its tet ids
  // and, per pixel, the bit set of the batch entries the pixel hit).  Round k takes entries [n c, n c + n) with
  // n = kEntries, c = rounds - 1 - k.  Its first loads come before the pixel's, which they do not depend on.
  const int64_t unit_at = (int64_t)u.tile * u.subs + u.sub;
  int nmax = (unit < n_units && RM_INDEX_OK(unit_at, RM_X_UNITS, 4)) ? __ldg(hit_counts + unit_at) : 0;
  const int64_t pix = (int64_t)u.y * rcam.image_width + u.x;
  float2 at_pixel = make_float2(0.5f, 0.5f);
  float logT = 0.f, sz = 0.f, sw = 0.f;
  float4 g4 = make_float4(0.f, 0.f, 0.f, 0.f);
  float gx2 = 0.f, gy2 = 0.f, gz = 0.f, gw = 0.f, gv = 0.f;
  if (u.inside) {
    if (jitter) at_pixel = __ldg(jitter + pix);
    logT = __ldg(out_img + pix).w;
    sz = __ldg(dist_img + 5 * pix + 2);
    sw = __ldg(dist_img + 5 * pix + 3);
    g4 = __ldg(g_img + pix);
    const float* gd = g_dist + 5 * pix;
    gx2 = 2.0f * __ldg(gd); gy2 = 2.0f * __ldg(gd + 1); gz = __ldg(gd + 2); gw = __ldg(gd + 3);
    gv = __ldg(gd + 4) * (1.0f / 3.0f);
  }
  const int64_t hbase = (int64_t)u.start * u.subs + (int64_t)u.sub * u.len;
  const int64_t mbase = hbase + 16 * unit_at;
  nmax = min(nmax, u.len);
  if (nmax > 0 && !(RM_INDEX_OK(hbase + nmax - 1, RM_X_HIT_IDS, 2) &&
                    RM_INDEX_OK(mbase + (nmax + kBatch - 1) / kBatch * kBatch - 1, RM_X_HIT_MASKS, 3)))
    nmax = 0;
  const int rounds = (nmax + kEntries - 1) / kEntries;
  const int max_rounds = max(rounds, __shfl_xor_sync(FULL, rounds, 16));

  // entry and row half this lane stages and sums in phase B
  const int ent = (PAIR ? lane : lane16) >> 1, part = lane16 & 1;
  int id_next = 0;         // tet id of `ent` in the round staged next
  unsigned bits_next = 0;  // this pixel's bits of that round
  int c = rounds - 1;      // the round that `fetch` reads
  int64_t id_at = hbase + (int64_t)c * kEntries + ent, mask_at = mbase + (int64_t)(PAIR ? c : c >> 1) * kBatch + lane16;
  // The places go down by steps; with those of a round from scratch each time, and the pixel's values before the hit
  // list's, 2M tets took 2.43 ms, not 2.36, and 21M 3.08, not 2.98.
  auto fetch = [&](bool whole) {
    bits_next = 0;
    if (c >= 0) {
      id_next = whole || c * kEntries + ent < nmax ? __ldg(hit_ids + id_at) : 0;
      bits_next = PAIR ? (unsigned)__ldg(hit_masks + mask_at) : ((unsigned)__ldg(hit_masks + mask_at) >> (kBwdBatch * (c & 1))) & 0xFFu;
      if (!RM_INDEX_OK(id_next, RM_X_TETS, 1)) id_next = 0;
      if (PAIR || !(c & 1)) mask_at -= kBatch;
      id_at -= kEntries;
      --c;
    }
  };
  auto stage = [&](int k) {
    if (k < rounds) {
      const float4* src = records + record_at(id_next) + 3 * part;
      float4* dst = staged + ent * kBwdStageStride + 3 * part;
#pragma unroll
      for (int q = 0; q < 3; ++q) cp_async16(dst + q, src + q);
    }
    cp_async_commit();
  };
  fetch(false);
  f3 d = {0.f, 0.f, 1.f};
  if (u.inside) d = ray_direction(rcam, (float)u.x + at_pixel.x, (float)u.y + at_pixel.y);
  stage(0);
  const float gr = g4.x, gg = g4.y, gb = g4.z, G = gr + gg + gb;
  float glogT = g4.w;
  sm.pixel[lane16][half][0] = make_float4(d.x, d.y, d.z, 1.0f);
  sm.pixel[lane16][half][1] = make_float4(gr, gg, gb, G);
  const float min_t = rcam.min_t;
  const Ray ray = make_ray(d);
  const float gx = 0.5f * gx2;
  // what phase A leaves of a hit: an entering distance te <= 0 is clamped and has no gradient
  auto leave = [&](int j, const Crossing& cr, float te, float g_enter, float g_exit, float a, float b, float w) {
    const float q_e = te > 0.0f ? -g_enter * cr.r_e : 0.0f, q_x = -g_exit * cr.r_x;
    rows[j].planes[lane16] = make_float4(q_e * cr.ue, q_e, q_x * cr.ux, q_x);
    rows[j].fields[lane16] = make_float4(a, b, w, w);
    reinterpret_cast<uint8_t*>(staged + j * kBwdStageStride + kFacesAt)[lane16] = (uint8_t)cr.faces;
  };
  float4* const faces_row = staged + ent * kBwdStageStride + kFacesAt;
  if (part == 0) *faces_row = make_float4(0.f, 0.f, 0.f, 0.f);
  for (int k = 0; k < max_rounds; ++k) {
    unsigned bits = bits_next;
    const int id = id_next;  // of the entry this lane sums
    fetch(true);
    cp_async_wait<0>();
    __syncwarp();

    // ---- phase A
    if constexpr (PAIR) {
      unsigned odd = bits ^ (bits >> 1);
      odd ^= odd >> 2;
      odd ^= odd >> 4;
      odd ^= odd >> 8;  // parity of the number of the pixel's entries from the last down to this one
      bits &= second ? ~odd : odd;
      while (__any_sync(FULL, bits != 0u)) {
        const int j = 31 - __clz(bits);  // -1 where no entry is left
        Crossing cr = {};
        float4 cg = make_float4(0.f, 0.f, 0.f, 0.f), cb = cg;
        if (j >= 0) {
          bits ^= 1u << j;
          const float4* rec = staged + j * kBwdStageStride;
          const float4 pl[4] = {rec[0], rec[1], rec[2], rec[3]};
          cg = rec[4];
          cb = rec[5];
          cr = slab_planes(pl, ray);
        }
        const float te = cr.ue - min_t, exit = cr.ux - min_t, enter = fmaxf(te, 0.0f), dt = exit - enter;
        const bool hit = cb.w * dt > 0.0f;
        const float tau = hit ? cb.w * dt : 0.0f, dens = hit ? cb.w : 0.0f;
        const float mid = (exit + enter) * 0.5f, m1 = hit ? dens * mid : 0.0f;
        const float o_tau = __shfl_xor_sync(FULL, tau, 16), o_dens = __shfl_xor_sync(FULL, dens, 16);
        const float o_m1 = __shfl_xor_sync(FULL, m1, 16);
        // the first lane's entry lies behind the second's and is undone before it
        const float logT1 = logT + (second ? o_tau : tau), logT2 = logT1 + (second ? tau : o_tau);
        const float sz1 = sz - (second ? o_dens : dens), sz2 = sz1 - (second ? dens : o_dens);
        const float sw1 = sw - (second ? o_m1 : m1), sw2 = sw1 - (second ? m1 : o_m1);
        const float gz1 = fmaf(second ? o_m1 : m1, gx2, gz), gw1 = fmaf(second ? o_dens : dens, gy2, gw);
        const float Tp = fast_exp(fminf(second ? logT2 : logT1, 46.0517f));
        const float g_m1 = fmaf(second ? sz2 : sz1, gx2, second ? gw1 : gw);
        const float g_m0 = fmaf(second ? sw2 : sw1, gy2, second ? gz1 : gz);
        const float X = exit + min_t, E = enter + min_t;
        const float gd = cg.x * d.x + cg.y * d.y + cg.z * d.z;
        const float oe = fmaf(E, gd, cg.w), ox = fmaf(X, gd, cg.w);
        float alpha = 0.f, w0 = 0.f, w1 = 0.f, slope = 0.f;
        if (hit) segment_weights(tau, alpha, w0, w1, slope);
        const float w = w0 + w1, gcb = gr * cb.x + gg * cb.y + gb * cb.z;
        const float up = hit ? fmaf(w, gcb, fmaf(w0, ox, w1 * oe) * G) * Tp : 0.0f;
        const float o_up = __shfl_xor_sync(FULL, up, 16), glogT1 = glogT + (second ? o_up : up);
        if (hit) {
          const float g_a = second ? -glogT1 : -glogT, TG = Tp * G, TC = Tp * gcb;
          const float g_ox = w0 * TG, g_oe = w1 * TG;
          const float g_tau = fmaf(TG * (oe - ox), slope, fmaf(fmaf(TG, ox, TC), alpha, g_a));
          const float gvd = gv * dens;
          const float b = fmaf(fmaf(2.0f, gvd, g_tau), dt, fmaf(g_m1, mid, g_m0));
          const float g_dt = fmaf(gvd, dens, g_tau * dens), g_mid = 0.5f * g_m1 * dens;
          const float g_exit = fmaf(g_ox, gd, g_mid) + g_dt, g_enter = fmaf(g_oe, gd, g_mid) - g_dt;
          leave(j, cr, te, g_enter, g_exit, fmaf(g_ox, X, g_oe * E), b, w * Tp);
        }
        logT = logT2;
        sz = sz2;
        sw = sw2;
        gz = fmaf(second ? m1 : o_m1, gx2, gz1);
        gw = fmaf(second ? dens : o_dens, gy2, gw1);
        glogT = glogT1 + (second ? up : o_up);
      }
    }
    while (!PAIR && bits) {
      const int j = 31 - __clz(bits);
      bits ^= 1u << j;
      const float4* rec = staged + j * kBwdStageStride;
      const float4 pl[4] = {rec[0], rec[1], rec[2], rec[3]};
      const float4 cg = rec[4], cb = rec[5];
      const Crossing cr = slab_planes(pl, ray);
      // A hit has entered before it leaves and leaves in front of the origin, so the leaving distance needs no
      // clamp.  (The forward pass found the optical depth positive with the same operations; the clamp only keeps
      // a disagreement from dividing by zero.)
      const float te = cr.ue - min_t, exit = cr.ux - min_t;
      const float enter = fmaxf(te, 0.0f), dens = cb.w;
      const float dt = exit - enter, tau = fmaxf(dens * dt, 1e-30f);
      const float X = cr.ux, E = fmaxf(cr.ue, min_t);
      const float gd = cg.x * d.x + cg.y * d.y + cg.z * d.z;
      const float oe = fmaf(E, gd, cg.w), ox = fmaf(X, gd, cg.w);
      float alpha, w0, w1, slope;
      segment_weights(tau, alpha, w0, w1, slope);
      // undo: state before this tet
      logT += tau;
      const float Tp = fast_exp(fminf(logT, 46.0517f));
      const float sum = exit + enter, m1x2 = dens * sum;  // twice the first moment
      // reverse of the state update
      sz -= dens;
      sw = fmaf(-0.5f, m1x2, sw);
      const float g_m1 = fmaf(sz, gx2, gw), g_m0 = fmaf(sw, gy2, gz);
      gw = fmaf(dens, gy2, gw);
      gz = fmaf(m1x2, gx, gz);
      const float gcb = gr * cb.x + gg * cb.y + gb * cb.z;  // colour of the tet against the upstream gradient
      // reverse of the segment integral
      const float TG = Tp * G, TC = Tp * gcb, w = w0 + w1;
      const float g_ox = w0 * TG, g_oe = w1 * TG;
      // d w0 / d tau = alpha + d phi / d tau, d w1 / d tau = -d phi / d tau, d phi / d tau = -slope
      const float g_tau = fmaf(TG * (oe - ox), slope, fmaf(fmaf(TG, ox, TC), alpha, -glogT));
      glogT += fmaf(w, TC, fmaf(g_ox, ox, g_oe * oe));
      const float gvd = gv * dens, half_m1 = 0.5f * g_m1;
      const float b = fmaf(fmaf(2.0f, gvd, g_tau), dt, fmaf(half_m1, sum, g_m0));
      const float g_dt = fmaf(gvd, dens, g_tau * dens), g_mid = half_m1 * dens;
      const float g_exit = fmaf(g_ox, gd, g_mid) + g_dt, g_enter = fmaf(g_oe, gd, g_mid) - g_dt;
      // planes: t = u - min_t, u = -D/den  =>  dt/dD = -1/den, dt/dn = -u/den d
      leave(j, cr, te, g_enter, g_exit, fmaf(g_ox, X, g_oe * E), b, w * Tp);
    }
    __syncwarp();
    // the entry's face bytes and the signs of its two planes' -D, before the copies of the next round and its phase A write there
    const float4 f4 = *faces_row;
    const float2 neg_d = reinterpret_cast<const float2*>(staged + ent * kBwdStageStride + 2 * part + 1)[1];
    const unsigned faces[4] = {__float_as_uint(f4.x), __float_as_uint(f4.y), __float_as_uint(f4.z), __float_as_uint(f4.w)};
    __syncwarp();
    if (!BEHIND && part == 0) *faces_row = make_float4(0.f, 0.f, 0.f, 0.f);
    stage(k + 1);

    // ---- phase B: part 0 sums planes 0 and 1, the colour gradient and the density, part 1 planes 2 and 3, the base colour and
    // the offset of the colour gradient; x, y and (z, the row's last)
    const BwdRow& row = rows[ent];
    const float2* const plane_pairs = reinterpret_cast<const float2*>(row.planes);
    const float2* const field_pairs = reinterpret_cast<const float2*>(row.fields) + part;
    const int side0 = neg_d.x < 0.0f ? 0 : 1, side1 = neg_d.y < 0.0f ? 0 : 1;  // entering (facing the camera) or leaving
    float x0 = 0.f, y0 = 0.f, x1 = 0.f, y1 = 0.f, xf = 0.f, yf = 0.f;
    float2 z0 = {0.f, 0.f}, z1 = z0, zf = z0;
    const unsigned plane0 = 0x01010101u << (4 * part), plane1 = 0x04040404u << (4 * part);
    const unsigned bits0 = plane0 << side0, bits1 = plane1 << side1;
#pragma unroll
    for (int p = 0; p < 16; ++p) {
      const unsigned byte = 0xFFu << (8 * (p & 3));
      const float4 dir = sm.pixel[p][half][0], con = sm.pixel[p][half][part];
      add_where(faces[p >> 2], bits0 & byte, plane_pairs[2 * p + side0], dir.x, dir.y, {dir.z, dir.w}, x0, y0, z0);
      add_where(faces[p >> 2], bits1 & byte, plane_pairs[2 * p + side1], dir.x, dir.y, {dir.z, dir.w}, x1, y1, z1);
      add_where(faces[p >> 2], byte, field_pairs[2 * p], con.x, con.y, {con.z, con.w}, xf, yf, zf);
    }
    const unsigned any = faces[0] | faces[1] | faces[2] | faces[3];
    const float last = __shfl_xor_sync(FULL, zf.y, 1);  // the density's sum belongs to the row of part 1, the offset's to part 0's
    if (any) {
      float4* out = reinterpret_cast<float4*>(grec + (int64_t)id * 24);
      if (any & bits0) atomicAdd(out + 2 * part, make_float4(x0, y0, z0.x, z0.y));
      if (any & bits1) atomicAdd(out + 2 * part + 1, make_float4(x1, y1, z1.x, z1.y));
      atomicAdd(out + 4 + part, make_float4(xf, yf, zf.x, last));
    }
    if constexpr (BEHIND) {  // hits that take a plane from its other side
      const unsigned other0 = bits0 ^ (3u * plane0), other1 = bits1 ^ (3u * plane1);
      if (any & (other0 | other1)) {
        float4 s0 = make_float4(0.f, 0.f, 0.f, 0.f), s1 = s0;
        auto add = [](float4& s, float2 v, float4 dir) {
          s = make_float4(fmaf(v.x, dir.x, s.x), fmaf(v.x, dir.y, s.y), fmaf(v.x, dir.z, s.z), s.w + v.y);
        };
#pragma unroll 1
        for (int p = 0; p < 16; ++p) {
          const unsigned face = reinterpret_cast<const uint8_t*>(faces_row)[p];
          if (face & other0) add(s0, plane_pairs[2 * p + (side0 ^ 1)], sm.pixel[p][half][0]);
          if (face & other1) add(s1, plane_pairs[2 * p + (side1 ^ 1)], sm.pixel[p][half][0]);
        }
        float4* out = reinterpret_cast<float4*>(grec + (int64_t)id * 24);
        if (any & other0) atomicAdd(out + 2 * part, s0);
        if (any & other1) atomicAdd(out + 2 * part + 1, s1);
      }
      __syncwarp();
      if (part == 0) *faces_row = make_float4(0.f, 0.f, 0.f, 0.f);
    }
  }
  cp_async_wait<0>();
}

// ----------------------------------------------------------------------------
// Backward of the constant-colour debug renderer, as the reference runs it
// (slang/alphablend_shader.slang:186-277, host side alphablend_tiled_slang.py:131-192): every pixel
// walks its tile list from its last contributor to the first; pairs with alpha < 1/255 are skipped
// (although the forward pass blended them); the state before a tet is recovered by undoing the update
// (transmittance by a division, replaced by 1 when 1 - alpha < 1e-3; distortion state with the weight
// (transmittance after the tet) * alpha); the derivatives of update_alpha_out and evaluate_tetra are taken
// at that recovered state.  A debug path: one lane per pixel, records read straight from global memory,
// gradients added to the record-gradient rows with 128-bit reductions (the reference issues 16 scalar
// atomics per hit); k_backward_finish then applies the chain rule to vertices and (r, g, b, density).
// ----------------------------------------------------------------------------
__device__ __forceinline__ float tukey_power_ladder_dx(float x, float p) {
  if (x == 0.0f) return 0.0f;
  const float q = fmaxf(fabsf(p - 1.0f), 1.0754944e-20f);
  return fabsf(p - 1.0f) / q * __powf(fabsf(x) / q + 1.0f, p - 1.0f);
}

__global__ void __launch_bounds__(kWarpsPerBlock * 32)
k_backward_cc(const int32_t* __restrict__ list, const int2* __restrict__ ranges, const float4* __restrict__ records,
              RmCamera rcam, const float4* __restrict__ out_img, const float4* __restrict__ dist_img,
              const int32_t* __restrict__ n_contrib, const float4* __restrict__ g_img,
              const float4* __restrict__ g_dist, float pre_multi, float ladder_p, float* __restrict__ grec, int subs,
              int64_t n_units) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int half = lane >> 4, lane16 = lane & 15;
  const int64_t unit = ((int64_t)blockIdx.x * kWarpsPerBlock + warp) * 2 + half;
  Unit u = make_unit(rcam, ranges, unit, n_units, subs, lane16);
  if (!u.inside) return;
  const int64_t pix = (int64_t)u.y * rcam.image_width + u.x;
  const f3 d = ray_direction(rcam, (float)u.x + 0.5f, (float)u.y + 0.5f);
  const Ray ray = make_ray(d);
  const float min_t = rcam.min_t;
  float4 st = __ldg(out_img + pix);   // r, g, b, transmittance
  float4 ds = __ldg(dist_img + pix);  // distortion state x, y, z, w
  float4 gi = __ldg(g_img + pix);
  float4 gd = __ldg(g_dist + pix);
  const int last = min(__ldg(n_contrib + pix), u.len);
  for (int j = last - 1; j >= 0; --j) {
    const int id = __ldg(list + u.start + j);
    if (!RM_INDEX_OK(id, RM_X_TETS, 7)) continue;
    const float4* rec = records + record_at(id);
    if (__ldg(rec + kLinesAt).y == never_seen()) continue;  // nothing else of this record is written
    const float4 pl[4] = {__ldg(rec), __ldg(rec + 1), __ldg(rec + 2), __ldg(rec + 3)};
    Eval ev;
    const float4 cb = __ldg(rec + 5);  // r, g, b, density
    if (!slab_test(pl, ray, min_t, cb.w, ev)) continue;  // no optical depth: alpha below 1/255, skipped too
    const Crossing cr = slab_planes(pl, ray);
    const float dens = cb.w;
    const float ex = __expf(-dens * ev.dt);
    const float a = fminf(fmaxf(1.0f - ex, 0.0f), 1.0f);
    if (a < 1.0f / 255.0f) continue;
    const float m = tukey_power_ladder(ev.enter * pre_multi, ladder_p);
    // undo
    const float w_u = st.w * a;
    const float Tp = (1.0f - a < 1e-3f) ? 1.0f : st.w / (1.0f - a);
    st.x -= a * cb.x * Tp;
    st.y -= a * cb.y * Tp;
    st.z -= a * cb.z * Tp;
    st.w = Tp;
    ds.z -= w_u;
    ds.w -= w_u * m;
    ds.x -= 2.0f * w_u * m * ds.z;
    ds.y -= 2.0f * w_u * ds.w;
    // reverse of the update at the recovered state
    const float weight = Tp * a;
    const float gcx = gi.x * Tp, gcy = gi.y * Tp, gcz = gi.z * Tp;
    float g_T = a * (gi.x * cb.x + gi.y * cb.y + gi.z * cb.z) + gi.w * (1.0f - a);
    float g_a = -gi.w * Tp;
    const float g_weight = gd.x * 2.0f * m * ds.z + gd.y * 2.0f * ds.w + gd.z + gd.w * m;
    const float g_m = gd.x * 2.0f * weight * ds.z + gd.w * weight;
    gd.z = gd.z + gd.x * 2.0f * weight * m;
    gd.w = gd.w + gd.y * 2.0f * weight;
    g_T += g_weight * a;
    g_a += g_weight * Tp;
    gi.w = g_T;
    float g_enter = g_m * tukey_power_ladder_dx(ev.enter * pre_multi, ladder_p) * pre_multi;
    // reverse of evaluate_tetra
    const float g_alpha = g_a + gcx * cb.x + gcy * cb.y + gcz * cb.z;
    const float inner = 1.0f - ex;
    const float g_tau = (inner > 0.0f && inner < 1.0f) ? g_alpha * ex : 0.0f;
    const float g_dt = g_tau * dens;
    float g_tx = 0.0f;
    if (ev.dt > 0.0f) { g_tx = g_dt; g_enter -= g_dt; }
    const float g_te = ev.te > 0.0f ? g_enter : 0.0f;
    float4* row = reinterpret_cast<float4*>(grec + (int64_t)id * 24);
    if (g_te != 0.0f) {
      const float q = -g_te * cr.r_e, uq = q * cr.ue;
      atomicAdd(row + __ffs(cr.faces & 0x55u) / 2, make_float4(uq * d.x, uq * d.y, uq * d.z, q));
    }
    if (g_tx != 0.0f) {
      const float q = -g_tx * cr.r_x, uq = q * cr.ux;
      atomicAdd(row + __ffs(cr.faces & 0xAAu) / 2 - 1, make_float4(uq * d.x, uq * d.y, uq * d.z, q));
    }
    atomicAdd(row + 5, make_float4(gcx * a, gcy * a, gcz * a, g_tau * ev.dt));
  }
}

// Clears the record-gradient rows (6 float4 each) of the tets flagged by the forward pass, and the vertex gradients.  Bound by its
// stores: the lanes of a warp clear the rows on its list side by side (four rows a thread by itself: 6.7M tets 76 us, now 47).
constexpr int kClearThreads = 256;
__global__ void __launch_bounds__(kClearThreads)
k_clear_flagged_rows(const uint8_t* __restrict__ tet_flags, int64_t T, float4* __restrict__ grec, float* __restrict__ vgrad,
                     int64_t n_vgrad) {
  after_previous();
  // four tets and four floats per thread: one 32-bit load of the flags
  const int64_t g4 = ((int64_t)blockIdx.x * kClearThreads + threadIdx.x) * 4;
  if (g4 + 4 <= n_vgrad && (reinterpret_cast<uintptr_t>(vgrad) & 15) == 0) {
    *reinterpret_cast<float4*>(vgrad + g4) = make_float4(0.f, 0.f, 0.f, 0.f);
  } else {
    for (int k = 0; k < 4 && g4 + k < n_vgrad; ++k) vgrad[g4 + k] = 0.0f;
  }
  uint32_t f4 = 0;
  if (g4 + 4 <= T && (reinterpret_cast<uintptr_t>(tet_flags) & 3) == 0) {
    f4 = *reinterpret_cast<const uint32_t*>(tet_flags + g4);
  } else {
    for (int k = 0; k < 4 && g4 + k < T; ++k) f4 |= (uint32_t)(tet_flags[g4 + k] != 0) << (8 * k);
  }
  // the warp lists its flagged tets and clears their rows side by side
  __shared__ uint8_t lists[kClearThreads * 4];
  const int lane = threadIdx.x & 31;
  uint8_t* const list = lists + 4 * (threadIdx.x & ~31u);
  int n = 0;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const bool on = (f4 >> (8 * k)) & 0xFFu;
    const unsigned m = __ballot_sync(0xffffffffu, on);
    if (on) list[n + __popc(m & ((1u << lane) - 1u))] = (uint8_t)(4 * lane + k);
    n += __popc(m);
  }
  __syncwarp();
  float4* const rows = grec + 6 * (g4 - 4 * lane);
  for (int i = lane; i < 6 * n; i += 32) {
    const int row = i / 6;
    rows[6 * list[row] + (i - 6 * row)] = make_float4(0.f, 0.f, 0.f, 0.f);
  }
}

// Chain rule from record gradients to vertices and cell values for tets [t_begin, T).  A warp looks through the flags of PER
// tets per lane and lists the flagged ones; a lane then takes one of the list.  Bound by the chain flag -> row and vertex ids ->
// vertices and by the atomics, on which all lanes of a warp are with a list, 20 of 32 with a tet per lane.  Warps wait for
// nobody: a list and rows of the whole block of 64 threads, PER = 4, cost meshes with a gradient in every tet more than a
// thread per tet did (1.05M 92.5 us -> 94.5, 2M in random order 168 -> 175; now 90.5 and 171).  Scenes with a thread per tet in
// blocks of 256: 2M 78 us, 6.7M 252, 21M 595; with lists 62, 187 and 353; with two reductions a vertex for three 54 and 162, and
// another view of the 21M scene 548 -> 494.
constexpr int kFinishThreads = 64;

template <int PER>
__global__ void __launch_bounds__(kFinishThreads)
k_backward_finish(const int32_t* __restrict__ indices, const float* __restrict__ vertices,
                  const float* __restrict__ cell, int64_t t_begin, int64_t T, RmCamera rcam,
                  const float4* __restrict__ grec, const uint8_t* __restrict__ tet_flags, float* __restrict__ vgrad,
                  float* __restrict__ cgrad) {
  // the cell-value gradient rows of a warp's tets (7 floats per tet, zero without a gradient) leave through shared memory as
  // contiguous 16-byte stores
  constexpr int kTets = 32 * PER;
  __shared__ __align__(16) float all_rows[kFinishThreads * PER * 7];
  __shared__ uint8_t lists[kFinishThreads * PER];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t g0 = t_begin + ((int64_t)blockIdx.x * kFinishThreads + 32 * warp) * PER;
  float* const rows = all_rows + warp * kTets * 7;
  uint8_t* const list = lists + warp * kTets;
  bool on[PER];
#pragma unroll
  for (int k = 0; k < PER; ++k) {
    const int64_t g = g0 + 32 * k + lane;
    on[k] = g < T && tet_flags[g];
  }
  for (int i = lane; i < kTets * 7 / 4; i += 32) reinterpret_cast<float4*>(rows)[i] = make_float4(0.f, 0.f, 0.f, 0.f);
  int n = 0;
#pragma unroll
  for (int k = 0; k < PER; ++k) {
    const unsigned m = __ballot_sync(0xffffffffu, on[k]);
    if (on[k]) list[n + __popc(m & ((1u << lane) - 1u))] = (uint8_t)(32 * k + lane);
    n += __popc(m);
  }
  __syncwarp();
  for (int i = lane; i < n; i += 32) {
    const int local = list[i];
    const int64_t g = g0 + local;
    float* co = rows + 7 * local;
    // the vertex ids travel with the gradient row: one dependent round trip less before the vertex gathers
    int4 id = __ldg(reinterpret_cast<const int4*>(indices) + g);
    float4 q[6];
    bool any = false;
#pragma unroll
    for (int k = 0; k < 6; ++k) {
      q[k] = __ldg(grec + 6 * g + k);
      any = any || q[k].x != 0.f || q[k].y != 0.f || q[k].z != 0.f || q[k].w != 0.f;
    }
    if (!any) continue;
    f3 cam = {__ldg(rcam.cam_pos), __ldg(rcam.cam_pos + 1), __ldg(rcam.cam_pos + 2)};
    if (!(RM_INDEX_OK(id.x, RM_X_VERTS, 5) && RM_INDEX_OK(id.y, RM_X_VERTS, 5) && RM_INDEX_OK(id.z, RM_X_VERTS, 5) &&
          RM_INDEX_OK(id.w, RM_X_VERTS, 5)))
      id = make_int4(0, 0, 0, 0);
    const int vid[4] = {id.x, id.y, id.z, id.w};
    f3 v[4] = {load3(vertices, id.x), load3(vertices, id.y), load3(vertices, id.z), load3(vertices, id.w)};
    PlaneSetup p;
    make_planes(v, cam, p);
    f3 gvv[4] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}, {0, 0, 0}};
  #pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int b = i == 3 ? 1 : 0;
      const int e1 = i < 2 ? 1 : 2;
      const int e2 = i == 0 ? 2 : 3;
      const float gD = q[i].w;
      f3 g_n = {q[i].x, q[i].y, q[i].z};
      g_n = g_n + (v[b] - cam) * (-gD);  // D = -n.(b - cam)
      f3 g_b = p.n[i] * (-gD);
      f3 g_raw = g_n * p.sgn[i];
      f3 E1 = v[e1] - v[b], E2 = v[e2] - v[b];
      f3 g_e1 = cross(E2, g_raw);
      f3 g_e2 = cross(g_raw, E1);
      gvv[e1] = gvv[e1] + g_e1;
      gvv[e2] = gvv[e2] + g_e2;
      gvv[b] = gvv[b] + g_b - g_e1 - g_e2;
    }
    const float* c = cell + 7 * g;
    f3 grd = {__ldg(c + 4), __ldg(c + 5), __ldg(c + 6)};
    const float gs0 = q[4].w;
    f3 g_grd = {q[4].x, q[4].y, q[4].z};
    g_grd = g_grd + (cam - v[0]) * gs0;  // s0 = grd.(cam - v0)
    gvv[0] = gvv[0] - grd * gs0;
  #pragma unroll
    for (int k = 0; k < 4; ++k) {
      // the two of a vertex's three floats that begin on 8 bytes in one reduction
      float* vp = vgrad + 3 * (int64_t)vid[k];
      const bool late = reinterpret_cast<uintptr_t>(vp) & 4;
      atomicAdd(reinterpret_cast<float2*>(vp + (late ? 1 : 0)), late ? make_float2(gvv[k].y, gvv[k].z) : make_float2(gvv[k].x, gvv[k].y));
      atomicAdd(vp + (late ? 0 : 2), late ? gvv[k].x : gvv[k].z);
    }
    co[0] = __ldg(c) > 0.0f ? q[5].w : 0.0f;
    co[1] = q[5].x;
    co[2] = q[5].y;
    co[3] = q[5].z;
    co[4] = g_grd.x;
    co[5] = g_grd.y;
    co[6] = g_grd.z;
  }
  __syncwarp();
  const int n_rows = (int)min((int64_t)kTets, T - g0);
  float* dst = cgrad + 7 * g0;
  if (n_rows == kTets && (reinterpret_cast<uintptr_t>(dst) & 15) == 0) {
    for (int i = lane; i < kTets * 7 / 4; i += 32)
      reinterpret_cast<float4*>(dst)[i] = reinterpret_cast<const float4*>(rows)[i];
  } else {
    for (int i = lane; i < n_rows * 7; i += 32) dst[i] = rows[i];
  }
}

// ----------------------------------------------------------------------------
// Distortion loss: mean over the pixels of max(0, (d0 - d1 + d4) / max(d2^2, 1e-6)), utils/train_util.py:58-62.
// One pass over the moments and a fixed-order sum of at most RM_LOSS_PARTIALS block sums, where torch takes nine
// kernels; bound by HBM for a large frame (20 bytes per pixel), by the two launches for a small one.
// A NaN passes both clamps, as in torch (fmaxf would drop it): the loss of a frame that has diverged shows it.
// ----------------------------------------------------------------------------
constexpr int kLossThreads = 256;
__device__ __forceinline__ float at_least(float x, float low) { return x < low ? low : x; }

__device__ __forceinline__ float block_sum(float v) {  // valid in thread 0
  __shared__ float s[kLossThreads / 32];
#pragma unroll
  for (int o = 16; o >= 1; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0) s[threadIdx.x >> 5] = v;
  __syncthreads();
  float t = 0.0f;
  if (threadIdx.x == 0) {
#pragma unroll
    for (int k = 0; k < kLossThreads / 32; ++k) t += s[k];
  }
  return t;
}

__global__ void __launch_bounds__(kLossThreads)
k_distortion_loss(const float* __restrict__ dist, int64_t n, float* __restrict__ partials) {
  after_previous();
  float sum = 0.0f;
  for (int64_t i = (int64_t)blockIdx.x * kLossThreads + threadIdx.x; i < n; i += (int64_t)gridDim.x * kLossThreads) {
    const float* d = dist + 5 * i;
    const float d2 = __ldg(d + 2);
    sum += at_least(((__ldg(d) - __ldg(d + 1)) + __ldg(d + 4)) / at_least(d2 * d2, 1e-6f), 0.0f);
  }
  const float t = block_sum(sum);
  if (threadIdx.x == 0) partials[blockIdx.x] = t;
}
__global__ void __launch_bounds__(kLossThreads)
k_distortion_loss_mean(const float* partials, int n_partials, int64_t n, float* __restrict__ loss) {
  after_previous();
  float sum = 0.0f;
  for (int i = threadIdx.x; i < n_partials; i += kLossThreads) sum += partials[i];
  const float t = block_sum(sum);
  if (threadIdx.x == 0) *loss = t / (float)n;
}

__global__ void __launch_bounds__(kLossThreads)
k_distortion_loss_backward(const float* __restrict__ dist, int64_t n, const float* __restrict__ g_loss,
                           float* __restrict__ g_dist) {
  __shared__ float rows[kLossThreads * 5];
  const int64_t first = (int64_t)blockIdx.x * kLossThreads;
  const int count = (int)min((int64_t)kLossThreads, n - first);
  for (int k = threadIdx.x; k < 5 * count; k += kLossThreads) rows[k] = __ldg(dist + 5 * first + k);
  __syncthreads();
  if (threadIdx.x < count) {
    float* d = rows + 5 * threadIdx.x;
    const float a = (d[0] - d[1]) + d[4], d2 = d[2], sq = d2 * d2, den = at_least(sq, 1e-6f), q = a / den;
    // both clamps pass the gradient at their bounds
    const float g = q >= 0.0f ? __ldg(g_loss) / (float)n : 0.0f, g_a = g / den;
    d[0] = g_a;
    d[1] = -g_a;
    d[2] = 2.0f * d2 * (sq >= 1e-6f ? -g_a * q : 0.0f);
    d[3] = 0.0f;
    d[4] = g_a;
  }
  __syncthreads();
  for (int k = threadIdx.x; k < 5 * count; k += kLossThreads) g_dist[5 * first + k] = rows[k];
}

}  // namespace rm

int rm_launch_distortion_loss(const float* dist, int64_t n, float* partials, float* loss, cudaStream_t st) {
  const int64_t want = (n + 4 * rm::kLossThreads - 1) / (4 * rm::kLossThreads);  // four pixels per thread, or more
  const int blocks = (int)(want < RM_LOSS_PARTIALS ? want : RM_LOSS_PARTIALS);
  RmProfScope prof("k_distortion_loss(2 launches)", st);
  RM_CUDA_CHECK(rm_launch(rm::k_distortion_loss, blocks, rm::kLossThreads, 0, st, dist, n, partials));
  RM_CUDA_CHECK(rm_launch_behind(blocks, rm::k_distortion_loss_mean, 1, rm::kLossThreads, 0, st, partials, blocks, n, loss));
  return RM_OK;
}

int rm_launch_distortion_loss_backward(const float* dist, int64_t n, const float* g_loss, float* g_dist, cudaStream_t st) {
  RmProfScope prof("k_distortion_loss_backward", st);
  RM_CUDA_CHECK(rm_launch(rm::k_distortion_loss_backward, (unsigned)((n + rm::kLossThreads - 1) / rm::kLossThreads),
                          rm::kLossThreads, 0, st, dist, n, g_loss, g_dist));
  return RM_OK;
}

// ----------------------------------------------------------------------------
// host-side launchers used by rm_api.cu
// ----------------------------------------------------------------------------
static inline void unit_grid(const RmCamera* cam, int warps, int* subs, int64_t* n_units, unsigned* blocks) {
  int px = cam->tile_width * cam->tile_height;
  *subs = (px + 15) / 16;
  int64_t tiles = (int64_t)(cam->tile_row_end - cam->tile_row_begin) * cam->grid_width;
  *n_units = tiles * *subs;
  int64_t per_block = warps * 2;
  *blocks = (unsigned)((*n_units + per_block - 1) / per_block);
}

// Up to a million tets a thread per tet, beyond several: large meshes are scenes of which a view sees a part and 40 % is empty,
// and they have blocks enough for a thread to look at several tets.  Packing with a thread per tet (with lists): 13k tets 8.5 us
// (15), scenes of 2M 77 (60), 6.7M 300 (236), 21M 937 (735), the last two in random order 330 (275), 1054 (961).  Meshes that
// have a record of every tet lose little by it: 0.6M 43 (47), 1.05M 64 (68), 2M 111 (112), 6.7M 364 (349).
// Chain rule: 0.6M all with a gradient 57.7 (59.8), 1.05M such 90.4 (90.6), 2M such 158 (156), 6.7M such 514 (501), scenes of
// 0.6M 23 (25), 2M 62 (62), 6.7M 195 (187), 21M 385 (353).
constexpr int64_t kListedTets = 1000000;

int rm_launch_pack(const int32_t* indices, const float* vertices, const float* cell, int64_t T, int64_t V,
                   const RmCamera* cam, const int32_t* tiles_touched, float* records, uint8_t* clear_a, uint8_t* clear_b,
                   cudaStream_t st) {
  if (T == 0) return RM_OK;
  RmProfScope prof("k_pack_records", st);
  const int per = T > kListedTets ? 3 : 1;
  auto kernel = per == 3 ? rm::k_pack_records<3> : rm::k_pack_records<1>;
  const int64_t per_block = (int64_t)per * rm::kPackThreads;
  RM_CUDA_CHECK(rm_launch(kernel, (unsigned)((T + per_block - 1) / per_block), rm::kPackThreads, 0, st, indices, vertices, cell, T, V, *cam,
                          tiles_touched, reinterpret_cast<float4*>(records), clear_a, clear_b));
  return RM_OK;
}

// n_list: entries of all lists, or -1 where the caller does not know.
//
// How the units are dealt to warps, by how often they fill the half-warps that the chip holds at a time ("waves"):
//   up to 2:   pairs.  The time is that of the longest lists.
//   up to 8:   pairs if the lists have 64 entries on average; shorter ones do not fill its batches of 32 (13k tets:
//              57 us in place of 64 on 400 x 400 pixels, but 95 in place of 84 on 560 x 560).
//   more:      long first, a long list being one of three times the average.  Up to five times the result is the
//              same within 1 %; at 1.5, pairs take over so much of the work that its overhead shows.
constexpr int64_t kWave = 148 * 20 * 2;
static bool deal_by_pairs(int64_t n_units, int64_t tiles, int64_t n_list) {
  return n_units <= 2 * kWave || (n_units <= 8 * kWave && n_list >= 64 * tiles);
}

// Whether hull lines are copied past L1: where lists have 800 entries on average, those of the tiles that an SM walks at a time name
// more lines than L1 holds (28 KB beside the walks' shared memory, and a line of it for each sector), and filling it costs more than
// the hits save (forward, through L1 and past it, by average list: 3M tets of a scene, 300 x 300, 2742: 1049 us, 846; 6.7M, 600 x 600,
// 1634: 736, 627; 21M, 1080p, 1886: 2166, 2024; 6.7M, 1080p, 1083: 1518, 1501; 1.2M in clusters, 300 x 300, 909: 304, 291).  Short
// lists live of it (0.6M, 800 x 800, 230: 375, 414; 1.2M, 600 x 600, 415: 400, 459); between 650 and 880 it is the same.
// The line lies there for larger tiles too, where 4 or 16 units walk one list: 8 x 8, 1M tets, 640 x 640, 922: 388, 359; 320 x 320,
// 1524: 437, 412; 6.7M, 1080p, 1380: 1712, 1644; 0.6M, 800 x 800, 343: 404, 539; 16 x 16, 1.3M, 800 x 800, 1300: 949, 936; 6.7M, 1080p,
// 2203: 2419, 2321; 0.3M and 0.6M, 800 x 800, 544 and 660: 522 and 504, 613 and 641.
static bool lines_past_l1(int64_t tiles, int64_t n_list) { return n_list >= 800 * tiles; }

int rm_launch_forward(const int32_t* list, const int32_t* ranges, const float* records, const RmCamera* cam,
                      const float* jitter, float* out_img, float* dist_img, int32_t* n_contrib, const RmHitList* hits,
                      int64_t n_list, cudaStream_t st) {
  int subs;
  int64_t n_units;
  unsigned blocks;
  unit_grid(cam, rm::kWarpsPerBlock, &subs, &n_units, &blocks);
  if (n_units == 0) return RM_OK;
  const int64_t tiles = n_units / subs;
  const unsigned pair_blocks = (unsigned)((n_units + rm::kWarpsPerBlock - 1) / rm::kWarpsPerBlock);
  const int threads = rm::kWarpsPerBlock * 32;
  const size_t smem = rm::kWarpsPerBlock * sizeof(rm::FwdShared);
  const int2* tiles_list = reinterpret_cast<const int2*>(ranges);
  const float4* recs = reinterpret_cast<const float4*>(records);
  const float2* jit = reinterpret_cast<const float2*>(jitter);
  float4* img = reinterpret_cast<float4*>(out_img);
  const RmHitList h = hits ? *hits : RmHitList{nullptr, nullptr, nullptr, nullptr};
  RmProfScope prof("k_forward", st);
  if (n_units > 8 * kWave && n_list >= 0) {
    constexpr int warps = rm::kLongFirstWarps, long_blocks = 148 * 20 / warps;
    const int long_list = (int)std::min<int64_t>(3 * n_list / tiles, INT_MAX);
    blocks = (unsigned)((n_units + 2 * warps - 1) / (2 * warps));
    auto kernel = lines_past_l1(tiles, n_list) ? rm::k_forward_long_first<true> : rm::k_forward_long_first<false>;
    RM_CUDA_CHECK(rm_launch(kernel, blocks + long_blocks, warps * 32, warps * sizeof(rm::FwdShared), st, list, tiles_list, recs, *cam,
                            jit, img, dist_img, n_contrib, h.counts, h.ids, h.masks, h.tet_flags, subs, n_units, long_list,
                            long_blocks));
  } else {
    const bool pair = deal_by_pairs(n_units, tiles, n_list);
    auto kernel = !pair ? rm::k_forward<rm::kColor, false, false>
                  : lines_past_l1(tiles, n_list) ? rm::k_forward<rm::kColor, true, true> : rm::k_forward<rm::kColor, true, false>;
    RM_CUDA_CHECK(rm_launch(kernel, pair ? pair_blocks : blocks, threads, smem, st, list, tiles_list, recs, *cam, jit, img,
                            dist_img, n_contrib, h.counts, h.ids, h.masks, h.tet_flags, subs, n_units, 0.0f, 0.0f,
                            rm::StatsArgs{}));
  }
  return RM_OK;
}

int rm_launch_forward_constant_color(const int32_t* list, const int32_t* ranges, const float* records,
                                     const RmCamera* cam, float pre_multi, float ladder_p, float* out_img,
                                     float* dist_img, int32_t* n_contrib, int64_t n_list, cudaStream_t st) {
  int subs;
  int64_t n_units;
  unsigned blocks;
  unit_grid(cam, rm::kWarpsPerBlock, &subs, &n_units, &blocks);
  if (n_units == 0) return RM_OK;
  RmProfScope prof("k_forward<constant colour>", st);
  const bool pair = deal_by_pairs(n_units, n_units / subs, n_list);
  if (pair) blocks = (unsigned)((n_units + rm::kWarpsPerBlock - 1) / rm::kWarpsPerBlock);
  auto kernel = pair ? rm::k_forward<rm::kConstColor, true, false> : rm::k_forward<rm::kConstColor, false, false>;
  RM_CUDA_CHECK(rm_launch(kernel, blocks, rm::kWarpsPerBlock * 32, rm::kWarpsPerBlock * sizeof(rm::FwdShared), st, list,
                          reinterpret_cast<const int2*>(ranges), reinterpret_cast<const float4*>(records), *cam, nullptr,
                          reinterpret_cast<float4*>(out_img), dist_img, n_contrib, nullptr, nullptr, nullptr, nullptr, subs,
                          n_units, pre_multi, ladder_p, rm::StatsArgs{}));
  return RM_OK;
}

int rm_launch_backward_constant_color(const int32_t* list, const int32_t* ranges, const float* records,
                                      const RmCamera* cam, float pre_multi, float ladder_p, const float* out_img,
                                      const float* dist_img, const int32_t* n_contrib, const float* g_img,
                                      const float* g_dist, int64_t T, int64_t V, float* grec, uint8_t* tet_flags,
                                      float* vgrad, cudaStream_t st) {
  RM_CUDA_CHECK(cudaMemsetAsync(vgrad, 0, sizeof(float) * 3 * (size_t)V, st));
  if (T == 0) return RM_OK;
  // every tet may receive a gradient here (the forward pass of this renderer keeps no hit lists)
  RM_CUDA_CHECK(cudaMemsetAsync(grec, 0, sizeof(float) * 24 * (size_t)T, st));
  RM_CUDA_CHECK(cudaMemsetAsync(tet_flags, 1, (size_t)T, st));
  int subs;
  int64_t n_units;
  unsigned blocks;
  unit_grid(cam, rm::kWarpsPerBlock, &subs, &n_units, &blocks);
  if (n_units > 0) {
    RmProfScope prof("k_backward<constant colour>", st);
    RM_CUDA_CHECK(rm_launch(rm::k_backward_cc, blocks, rm::kWarpsPerBlock * 32, 0, st, list,
                            reinterpret_cast<const int2*>(ranges), reinterpret_cast<const float4*>(records), *cam,
                            reinterpret_cast<const float4*>(out_img), reinterpret_cast<const float4*>(dist_img), n_contrib,
                            reinterpret_cast<const float4*>(g_img), reinterpret_cast<const float4*>(g_dist),
                            pre_multi, ladder_p, grec, subs, n_units));
  }
  return RM_OK;
}

int rm_launch_tet_err(const int32_t* list, const int32_t* ranges, const float* records, const RmCamera* cam,
                      const float* pixel_err, const float* ssim_err, int64_t T, float* tet_err, int32_t* tet_count,
                      cudaStream_t st) {
  if (T == 0) return RM_OK;
  RM_CUDA_CHECK(cudaMemsetAsync(tet_err, 0, sizeof(float) * 16 * (size_t)T, st));
  RM_CUDA_CHECK(cudaMemsetAsync(tet_count, 0, sizeof(int32_t) * 2 * (size_t)T, st));
  int subs;
  int64_t n_units;
  unsigned blocks;
  constexpr int warps = rm::kFwdWarps<rm::kStats>;
  unit_grid(cam, warps, &subs, &n_units, &blocks);
  if (n_units == 0) return RM_OK;
  constexpr size_t smem = warps * sizeof(rm::StatsShared);
  RM_CUDA_CHECK(cudaFuncSetAttribute(rm::k_forward<rm::kStats, false, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)smem));
  RmProfScope prof("k_tet_err", st);
  RM_CUDA_CHECK(rm_launch(rm::k_forward<rm::kStats, false, false>, blocks, warps * 32, smem, st, list,
                          reinterpret_cast<const int2*>(ranges), reinterpret_cast<const float4*>(records), *cam, nullptr,
                          nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, subs, n_units, 0.0f, 0.0f,
                          rm::StatsArgs{pixel_err, ssim_err, tet_err, tet_count}));
  return RM_OK;
}

static int launch_backward_walk(const int32_t* ranges, const float* records, const RmCamera* cam, const float* jitter,
                                const float* out_img, const float* dist_img, const RmHitList* hits, const float* g_img,
                                const float* g_dist, float* grec, int64_t T, cudaStream_t st) {
  int subs;
  int64_t n_units;
  unsigned blocks;
  unit_grid(cam, rm::kBwdWarps<false>, &subs, &n_units, &blocks);
  if (n_units == 0) return RM_OK;
  // up to two waves of half-warps the longest hit lists set the time; beyond, the shuffles' cost shows (2M tets, 400 x 400:
  // 683 -> 662 us, 560 x 560: 1039 -> 1092 us)
  const bool pair = n_units <= 2 * kWave;
  const int warps = pair ? rm::kBwdWarps<true> : rm::kBwdWarps<false>;
  if (pair) blocks = (unsigned)((n_units + warps - 1) / warps);
  const size_t smem = warps * sizeof(rm::BwdShared);
  const bool behind = !(cam->min_t >= 0.0f);
  auto kernel = pair ? (behind ? rm::k_backward<true, true> : rm::k_backward<true, false>)
                     : (behind ? rm::k_backward<false, true> : rm::k_backward<false, false>);
  RM_CUDA_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  RmProfScope prof("k_backward", st);
  RM_CUDA_CHECK(rm_launch_behind(T, kernel, blocks, warps * 32, smem, st,
                                 reinterpret_cast<const int2*>(ranges), reinterpret_cast<const float4*>(records), *cam,
                                 reinterpret_cast<const float2*>(jitter), reinterpret_cast<const float4*>(out_img), dist_img,
                                 hits->counts, hits->ids, hits->masks, reinterpret_cast<const float4*>(g_img), g_dist, grec,
                                 subs, n_units));
  return RM_OK;
}

static int launch_clear(const RmHitList* hits, int64_t T, int64_t V, float* grec, float* vgrad, cudaStream_t st) {
  const int64_t n = (T > 3 * V ? T : 3 * V), per_block = 4 * rm::kClearThreads;
  if (n == 0) return RM_OK;
  RmProfScope prof("k_clear_flagged_rows", st);
  RM_CUDA_CHECK(rm_launch(rm::k_clear_flagged_rows, (unsigned)((n + per_block - 1) / per_block), rm::kClearThreads, 0, st,
                          hits->tet_flags, T, reinterpret_cast<float4*>(grec), vgrad, 3 * V));
  return RM_OK;
}

// Everything of the backward pass except the per-tet chain rule: clears vertices_grad and the
// record-gradient rows of flagged tets, then accumulates the record gradients.
int rm_launch_backward_integrate(const int32_t* ranges, const float* records, const RmCamera* cam, const float* jitter,
                                 const float* out_img, const float* dist_img, const RmHitList* hits, const float* g_img,
                                 const float* g_dist, int64_t T, int64_t V, float* grec, float* vgrad,
                                 cudaStream_t st) {
  int rc = launch_clear(hits, T, V, grec, vgrad, st);
  if (rc || T == 0) return rc;
  return launch_backward_walk(ranges, records, cam, jitter, out_img, dist_img, hits, g_img, g_dist, grec, T, st);
}

// The chain rule from record gradients to vertices and cell values for tets [t_begin, t_end).
int rm_launch_backward_finish(const int32_t* indices, const float* vertices, const float* cell, int64_t t_begin,
                              int64_t t_end, const RmCamera* cam, const float* grec, const RmHitList* hits,
                              float* vgrad, float* cgrad, cudaStream_t st) {
  if (t_end <= t_begin) return RM_OK;
  RmProfScope prof("k_backward_finish", st);
  const int64_t n = t_end - t_begin;
  const int per = n > kListedTets ? 3 : 1;
  auto kernel = per == 3 ? rm::k_backward_finish<3> : rm::k_backward_finish<1>;
  const int64_t per_block = (int64_t)per * rm::kFinishThreads;
  RM_CUDA_CHECK(rm_launch(kernel, (unsigned)((n + per_block - 1) / per_block), rm::kFinishThreads, 0, st, indices, vertices, cell,
                          t_begin, t_end, *cam, reinterpret_cast<const float4*>(grec), hits->tet_flags, vgrad, cgrad));
  return RM_OK;
}

// ----------------------------------------------------------------------------
// rm_backward_static_scratch: the backward pass for callers that may not
// allocate device memory.  Its only scratch, the per-tet record-gradient rows,
// lives in the file-scope device array below instead of a caller buffer.
// ----------------------------------------------------------------------------
#include <mutex>

static __device__ __align__(256) float g_static_grad_records[(size_t)RM_STATIC_SCRATCH_MAX_TETS * RM_GRAD_RECORD_FLOATS];

namespace {
constexpr int kMaxDevices = 64;
std::mutex g_static_mu;
float* g_static_addr[kMaxDevices] = {nullptr};
}  // namespace

extern "C" int rm_backward_static_scratch(const int32_t* sorted_tetra_idx, const int32_t* tile_ranges,
                                          const float* records, const RmCamera* cam, const float* ray_jitter,
                                          const float* output_img, const float* distortion_img,
                                          const int32_t* n_contributors, const RmHitList* hits,
                                          const float* grad_output_img,
                                          const float* grad_distortion_img, const int32_t* indices,
                                          const float* vertices, const float* cell_values, int64_t n_tets,
                                          int64_t n_vertices, float* vertices_grad, float* cell_values_grad,
                                          void* stream) {
  // the same host-side checks as rm_backward, before anything touches the device
  rm_clear_last_error();
  if (n_tets > RM_STATIC_SCRATCH_MAX_TETS) return RM_ERR_STATIC_SCRATCH;
  int rc = rm_check_cam(cam);
  if (rc) return rc;
  if (n_tets < 0 || n_vertices < 0) return RM_ERR_INVALID_ARG;
  if (!tile_ranges || !output_img || !distortion_img || !hits || !hits->counts || !hits->ids ||
      !hits->masks || !hits->tet_flags || !grad_output_img || !grad_distortion_img || !vertices_grad)
    return RM_ERR_INVALID_ARG;
  (void)sorted_tetra_idx;
  (void)n_contributors;
  if (n_tets > 0 && (!indices || !vertices || !cell_values || !cell_values_grad || !records))
    return RM_ERR_INVALID_ARG;
  if (!rm_aligned16(output_img) || !rm_aligned16(grad_output_img) || !rm_aligned16(records) || !rm_aligned16(indices))
    return RM_ERR_WORKSPACE;
  rc = rm_bind_device(vertices_grad);  // makes the device that owns the buffers current
  if (rc) return rc;
  // Set-up, once per device, with that device current: the array's name is a
  // host-side handle, the kernels need its device address.
  int dev = -1;
  RM_CUDA_CHECK(cudaGetDevice(&dev));
  if (dev < 0 || dev >= kMaxDevices) return RM_ERR_INVALID_ARG;
  float* scratch = nullptr;
  {
    std::lock_guard<std::mutex> lk(g_static_mu);
    if (!g_static_addr[dev]) {
      void* addr = nullptr;
      RM_CUDA_CHECK(cudaGetSymbolAddress(&addr, g_static_grad_records));
      g_static_addr[dev] = static_cast<float*>(addr);
    }
    scratch = g_static_addr[dev];
  }
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  // The array keeps the previous call's sums: clear the rows this call accumulates into.
  rc = launch_clear(hits, n_tets, n_vertices, scratch, vertices_grad, st);
  if (rc || n_tets == 0) return rc;
  rc = launch_backward_walk(tile_ranges, records, cam, ray_jitter, output_img, distortion_img, hits, grad_output_img,
                            grad_distortion_img, scratch, n_tets, st);
  if (rc) return rc;
  return rm_launch_backward_finish(indices, vertices, cell_values, 0, n_tets, cam, scratch, hits, vertices_grad, cell_values_grad,
                                   st);
}

// Bounds-checked build: extents of the caller-owned arrays of the integration stages (the entry points
// of these stages carry no array lengths) and the status word of this translation unit.
unsigned rm_bounds_status_raster() { return rm_take_bounds_status(); }
void rm_debug_extent_raster(int which, long long n) {
  if (which >= 0 && which < RM_X_COUNT) rm_set_extent(which, n, nullptr);
#ifdef RM_BOUNDS_CHECK
  cudaDeviceSynchronize();
#endif
}
