// Shared device/host helpers for the sm_100a rasterizer kernels.
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

#include "rm_b200.h"

#define RM_CUDA_CHECK(expr)                          \
  do {                                               \
    cudaError_t _e = (expr);                         \
    if (_e != cudaSuccess) {                         \
      rm_set_last_cuda_error(_e, __FILE__, __LINE__); \
      return RM_ERR_CUDA;                            \
    }                                                \
  } while (0)

void rm_set_last_cuda_error(cudaError_t e, const char* file, int line);
void rm_clear_last_error();
int rm_bind_device(const void* device_ptr);
// Host-side checks every entry point applies to its camera and to pointers it accesses with
// 128-bit loads or stores.
int rm_check_cam(const RmCamera* c);
static inline bool rm_aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

// Every kernel launch of the library is counted (rm_launch_count), so that a caller can state how
// many of this library's kernels ran inside a timed region.
void rm_count_launch();

// All launches go through these two, which return the launch's own error: what follows on a kernel that did not start would
// run on memory that nobody has written.
template <typename... P, typename... A>
cudaError_t rm_launch_config(bool behind, void (*kernel)(P...), unsigned blocks, unsigned threads, size_t smem, cudaStream_t st,
                             A... args) {
  rm_count_launch();
  cudaLaunchAttribute attribute = {};
  attribute.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attribute.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t config = {};
  config.gridDim = dim3(blocks);
  config.blockDim = dim3(threads);
  config.dynamicSmemBytes = smem;
  config.stream = st;
  config.attrs = &attribute;
  config.numAttrs = behind ? 1 : 0;
  return cudaLaunchKernelEx(&config, kernel, static_cast<P>(args)...);
}
template <typename... P, typename... A>
cudaError_t rm_launch(void (*kernel)(P...), unsigned blocks, unsigned threads, size_t smem, cudaStream_t st, A... args) {
  return rm_launch_config(false, kernel, blocks, threads, smem, st, args...);
}

// Launch of a kernel that begins with rm::after_previous(), behind a kernel that the same call of the library has launched on
// the same stream: its blocks are placed while the last blocks of that kernel still run, and wait there for its end.  Never for
// the first launch of a call, which may have to wait for copies and events of the caller's.  Only for `items` (tets or pairs)
// up to kFewItems, where the 2 to 3 us between the kernels count (60k tets, 203 x 317 pixels: frame 209 -> 194 us); the
// waiting blocks of larger grids hold back more than that (600k tets, 800 x 800: 687 -> 699 us).
constexpr int64_t kFewItems = 1 << 17;
template <typename... P, typename... A>
cudaError_t rm_launch_behind(int64_t items, void (*kernel)(P...), unsigned blocks, unsigned threads, size_t smem, cudaStream_t st,
                             A... args) {
  return rm_launch_config(items <= kFewItems, kernel, blocks, threads, smem, st, args...);
}

// Optional per-kernel timing (rm_profile_enable): a scope records a CUDA event
// pair on the launch stream around the launches it encloses.
void rm_prof_begin(const char* name, cudaStream_t st);
void rm_prof_end(cudaStream_t st);
struct RmProfScope {
  cudaStream_t st;
  RmProfScope(const char* name, cudaStream_t s) : st(s) { rm_prof_begin(name, s); }
  ~RmProfScope() { rm_prof_end(st); }
};

// ---------------------------------------------------------------------------
// Bounds-checked build (-DRM_BOUNDS_CHECK), used by the tests in place of a memory checker: every
// index that depends on data (list cursors, hit-list slots, ids read from lists, rows addressed by
// them) is tested against the extent of its array before the access; a violation sets a bit of a
// status word that rm_debug_bounds_status() returns and the access is skipped - nothing traps.  The
// extents are set by the host launchers before each launch.  In the normal build the macros vanish.
// ---------------------------------------------------------------------------
enum RmExtent {
  RM_X_LIST = 0,      // sorted_tetra_idx entries
  RM_X_TETS,          // records / record-gradient rows / tet_flags / per-tet outputs
  RM_X_VERTS,         // vertices
  RM_X_HIT_IDS,       // hit-list id slots
  RM_X_HIT_MASKS,     // hit-list mask slots
  RM_X_UNITS,         // hit-list counts
  RM_X_PAIRS,         // (region, tet) pairs / sorted region entries
  RM_X_CHUNKS,        // chunks of the level-2 list build
  RM_X_REGIONS,       // regions
  RM_X_TILES,         // tiles
  RM_X_COUNT
};
#ifdef RM_BOUNDS_CHECK
static __device__ long long g_rm_extent[RM_X_COUNT];
static __device__ unsigned g_rm_bounds_status;
// site: a small number naming the access, reported as bit (site & 31)
#define RM_INDEX_OK(i, which, site) rm_index_ok((long long)(i), g_rm_extent[which], (site))
static __device__ __forceinline__ bool rm_index_ok(long long i, long long n, int site) {
  if ((unsigned long long)i < (unsigned long long)n) return true;
  atomicOr(&g_rm_bounds_status, 1u << (site & 31));
  return false;
}
static inline void rm_set_extent(int which, long long n, cudaStream_t st) {
  cudaMemcpyToSymbolAsync(g_rm_extent, &n, sizeof(n), sizeof(long long) * (size_t)which, cudaMemcpyHostToDevice, st);
}
static inline unsigned rm_take_bounds_status() {
  unsigned v = 0, z = 0;
  cudaDeviceSynchronize();
  cudaMemcpyFromSymbol(&v, g_rm_bounds_status, sizeof(v));
  cudaMemcpyToSymbol(g_rm_bounds_status, &z, sizeof(z));
  return v;
}
#else
#define RM_INDEX_OK(i, which, site) true
static inline void rm_set_extent(int, long long, cudaStream_t) {}
static inline unsigned rm_take_bounds_status() { return 0; }
#endif
unsigned rm_bounds_status_raster();
unsigned rm_bounds_status_binning();
unsigned rm_take_recounted();

namespace rm {

// First statement of every thread of a kernel that may be launched with rm_launch_behind, or in front of one, before any
// access to memory: lets the next kernel's blocks be placed as soon as all of this one's are, and waits until the kernel
// before has ended and what it wrote can be seen.  The wait returns at once after an ordinary launch.
// A kernel that is launched behind another is there while the kernels before it in the chain still write.  What those
// write it reads with plain loads from pointers without __restrict__: __ldg, and const __restrict__, tell the compiler that
// the data stay the same for as long as the kernel is there, which lets it move the loads in front of the wait and serve
// them from a cache that is not kept coherent.
__device__ __forceinline__ void after_previous() {
  asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
  asm volatile("griddepcontrol.wait;\n" ::: "memory");
}

constexpr int kRecordFloats = RM_RECORD_FLOATS;

// Camera in registers / shared memory.  Loaded from the device arrays of
// RmCamera so that the host never has to read them back.
struct DevCam {
  float W[16];
  float K[9];
  float pos[3];
  float dist[4];
  int H, Wd, type;
  float min_t;
  int tile_h, tile_w, grid_h, grid_w;
  int row0, row1;
  float inv_tile_h, inv_tile_w;  // rounded
};

// By the first warp of a block into shared memory; the caller's next barrier makes it visible.
__device__ __forceinline__ void load_cam_shared(const RmCamera& c, DevCam& d) {
  static_assert(sizeof(DevCam) >= 32 * sizeof(float) && offsetof(DevCam, K) == 64 && offsetof(DevCam, pos) == 100 &&
                    offsetof(DevCam, dist) == 112,
                "the device arrays are the first 32 floats");
  const int i = threadIdx.x;
  if (i < 32) {
    reinterpret_cast<float*>(&d)[i] = i < 16   ? __ldg(c.world_view_transform + i)
                                      : i < 25 ? __ldg(c.K + i - 16)
                                      : i < 28 ? __ldg(c.cam_pos + i - 25)
                                               : __ldg(c.distortion_params + i - 28);
  }
  if (i == 0) {
    d.H = c.image_height;
    d.Wd = c.image_width;
    d.type = c.camera_type;
    d.min_t = c.min_t;
    d.tile_h = c.tile_height;
    d.tile_w = c.tile_width;
    d.grid_h = c.grid_height;
    d.grid_w = c.grid_width;
    d.row0 = c.tile_row_begin;
    d.row1 = c.tile_row_end;
    d.inv_tile_h = 1.0f / float(c.tile_height);
    d.inv_tile_w = 1.0f / float(c.tile_width);
  }
}

// The hardware's approximation with denormals flushed; the plain forms (__fdividef, __frcp_rn) rescale around denormal
// operands.
__device__ __forceinline__ float fast_rcp(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

struct f3 {
  float x, y, z;
};
__device__ __forceinline__ f3 operator+(f3 a, f3 b) { return {a.x + b.x, a.y + b.y, a.z + b.z}; }
__device__ __forceinline__ f3 operator-(f3 a, f3 b) { return {a.x - b.x, a.y - b.y, a.z - b.z}; }
__device__ __forceinline__ f3 operator*(f3 a, float s) { return {a.x * s, a.y * s, a.z * s}; }
__device__ __forceinline__ f3 operator-(f3 a) { return {-a.x, -a.y, -a.z}; }
__device__ __forceinline__ float dot(f3 a, f3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
__device__ __forceinline__ f3 cross(f3 a, f3 b) {
  return {a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x};
}
__device__ __forceinline__ f3 load3(const float* p, int64_t i) {
  return {__ldg(p + 3 * i), __ldg(p + 3 * i + 1), __ldg(p + 3 * i + 2)};
}

struct d3 {
  double x, y, z;
};
__device__ __forceinline__ d3 operator+(d3 a, d3 b) { return {a.x + b.x, a.y + b.y, a.z + b.z}; }
__device__ __forceinline__ d3 operator-(d3 a, d3 b) { return {a.x - b.x, a.y - b.y, a.z - b.z}; }
__device__ __forceinline__ d3 operator*(d3 a, double s) { return {a.x * s, a.y * s, a.z * s}; }
__device__ __forceinline__ double dot(d3 a, d3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
__device__ __forceinline__ d3 cross(d3 a, d3 b) {
  return {a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x};
}

// Order-preserving map float -> uint32 (slang/tile_shader.slang:18-47).
__device__ __forceinline__ uint32_t float2sortable_key(float v) {
  uint32_t bits = __float_as_uint(v);
  return (bits & 0x80000000u) ? ~bits : (bits ^ 0x80000000u);
}

}  // namespace rm
