// Host path of the rasterizer for PyTorch callers: allocation of outputs and workspaces, the calls into the C ABI
// (include/rm_b200.h) and the one host synchronisation of a frame, in native code.  A small frame is bound by the
// host: with the same steps in Python (about 25 torch.empty calls, 9 ctypes calls, the checks between them) a
// 13k-tet, 128 x 128 training view took 0.8 ms of which the GPU was busy for 0.4.
//
// The library is opened by path (bind), so that this module drives whichever build of it the package has loaded.

#include <ATen/ATen.h>
#include <ATen/cuda/CUDAContext.h>
#include <ATen/cuda/CUDAEvent.h>
#include <c10/cuda/CUDAGuard.h>
#include <dlfcn.h>
#include <torch/extension.h>

#include "rm_b200.h"

namespace py = pybind11;
using at::Tensor;

namespace {

#define RM_FUNCTIONS(X)                                                                                              \
  X(rm_strerror) X(rm_bin_workspace_bytes) X(rm_list_scratch_bytes) X(rm_project_and_bin_visible) X(rm_build_tile_lists) \
  X(rm_pack_records_and_clear) X(rm_forward_sized) X(rm_backward) X(rm_vertex_backward) X(rm_tet_err) X(rm_activate_output)  \
  X(rm_distortion_loss) X(rm_distortion_loss_backward) X(rm_debug_bounds_checked)         \
  X(rm_debug_set_extent)
#define DECLARE(name) decltype(&::name) name = nullptr;
struct Library {
  RM_FUNCTIONS(DECLARE)
  bool checked = false;
} lib;

void bind(const std::string& path) {
  void* h = dlopen(path.c_str(), RTLD_NOW | RTLD_LOCAL);
  if (!h) throw std::runtime_error(std::string("rm_b200: ") + dlerror());
#define RESOLVE(name)                                                                                  \
  lib.name = reinterpret_cast<decltype(lib.name)>(dlsym(h, #name));                                    \
  if (!lib.name) throw std::runtime_error("rm_b200: " #name " is missing from " + path);
  RM_FUNCTIONS(RESOLVE)
  lib.checked = lib.rm_debug_bounds_checked() != 0;
}

void check(int rc) {
  if (rc) throw std::runtime_error(std::string("rm_b200: ") + lib.rm_strerror(rc) + " (code " + std::to_string(rc) + ")");
}

const RmCamera* camera(uintptr_t address) { return reinterpret_cast<const RmCamera*>(address); }
void* stream_of(const Tensor& t) { return c10::cuda::getCurrentCUDAStream(t.device().index()).stream(); }

template <typename T>
T* ptr(const Tensor& t) {
  return static_cast<T*>(t.data_ptr());
}
template <typename T>
T* ptr(const c10::optional<Tensor>& t) {
  return t.has_value() ? static_cast<T*>(t->data_ptr()) : nullptr;
}

Tensor empty(at::IntArrayRef size, at::ScalarType type, const at::Device& device) {
  return at::empty(size, at::TensorOptions().dtype(type).device(device));
}
Tensor i32(const Tensor& t) { return t.scalar_type() == at::kInt ? t.contiguous() : t.contiguous().to(at::kInt); }
Tensor f32(const Tensor& t) {
  const Tensor d = t.requires_grad() ? t.detach() : t;
  return d.scalar_type() == at::kFloat ? d.contiguous() : d.contiguous().to(at::kFloat);
}
void require_cuda(const Tensor& t, const char* name) {
  if (!t.is_cuda()) throw std::runtime_error(std::string(name) + " must be a CUDA tensor (the rasterizer has no CPU path)");
}
void extents(std::initializer_list<std::pair<int, int64_t>> list) {  // bounds-checked build only
  if (lib.checked)
    for (auto& e : list) lib.rm_debug_set_extent(e.first, e.second);
}
enum { kList, kTets, kVerts, kHitIds, kHitMasks, kUnits };

// The camera dictionary (data/camera.py:72-91 plus the tile fields of utils/train_util.py:30-37), or any object with its
// subscripts and its get, as an RmCamera, with the device tensors it points at.
struct Camera {
  RmCamera c;
  Tensor keep[4];
  bool band_rows_only;

  Camera(const py::object& d, const at::Device& device, const py::object& tile_rows) {
    static const char* names[4] = {"world_view_transform", "K", "cam_pos", "distortion_params"};
    static const int64_t sizes[4] = {16, 9, 3, 4};
    const float** slots[4] = {&c.world_view_transform, &c.K, &c.cam_pos, &c.distortion_params};
    for (int i = 0; i < 4; ++i) {
      py::object o = d[names[i]];
      if (!THPVariable_Check(o.ptr())) o = py::module_::import("torch").attr("as_tensor")(o);
      Tensor t = THPVariable_Unpack(o.ptr());
      if (t.device() != device || t.scalar_type() != at::kFloat) t = t.to(device, at::kFloat);
      keep[i] = t.contiguous();
      if (keep[i].numel() != sizes[i]) throw py::value_error(std::string("camera: ") + names[i] + " has the wrong size");
      *slots[i] = ptr<float>(keep[i]);
    }
    auto integer = [&](const char* k) { return py::int_(py::object(d[k])).cast<int32_t>(); };
    auto real = [&](const char* k) { return (float)py::float_(py::object(d[k])).cast<double>(); };
    c.image_height = integer("image_height");
    c.image_width = integer("image_width");
    c.camera_type = integer("camera_type");
    c.fovy = real("fovy");
    c.fovx = real("fovx");
    c.min_t = real("min_t");
    c.tile_height = integer("tile_height");
    c.tile_width = integer("tile_width");
    c.grid_height = integer("grid_height");
    c.grid_width = integer("grid_width");
    c.tile_row_begin = 0;
    c.tile_row_end = c.grid_height;
    const py::object get = d.attr("get");
    py::object rows = !tile_rows.is_none() ? tile_rows : get("tile_rows", py::none());
    if (!rows.is_none()) {
      c.tile_row_begin = py::int_(py::object(rows[py::int_(0)])).cast<int32_t>();
      c.tile_row_end = py::int_(py::object(rows[py::int_(1)])).cast<int32_t>();
    }
    // a band-restricted call zero-fills the image rows outside its band unless the caller reads the band only
    band_rows_only = py::bool_(get("band_rows_only", false)).cast<bool>();
  }
};

// A copy of a frame's info block in page-locked memory, which the device has written once the stream has passed `written`.  The
// memory goes back only after that, also where a frame is given up in between: it would otherwise be somebody else's by then.
struct PendingInfo {
  Tensor block;
  at::cuda::CUDAEvent written;
  c10::cuda::CUDAStream stream;
  bool arrived = false;

  explicit PendingInfo(c10::cuda::CUDAStream s)
      : block(at::empty({3}, at::TensorOptions().dtype(at::kLong).pinned_memory(true))), stream(s) {}
  ~PendingInfo() {
    if (!arrived) cudaStreamSynchronize(stream.stream());
  }
  void record() { written.record(stream); }
  // The one host synchronisation of a frame: (list entries, region pairs, visible tets, status bits).  What was enqueued behind
  // the info block is not waited for.
  std::tuple<int64_t, int64_t, int64_t, int64_t> wait() {
    if (!arrived) written.synchronize();
    arrived = true;
    const RmBinInfo* r = ptr<RmBinInfo>(block);
    return {r->n_keys, r->n_region_keys, r->n_visible, r->status};
  }
};

// Stage 1 and tile populations.  Returns ((indices, vertices, tiles_touched, rect, vs_tetra, circumcenter, tile_ranges,
// info, workspace, visible), host copy of info if asked for).
std::tuple<std::vector<Tensor>, std::unique_ptr<PendingInfo>> project_and_bin(const Tensor& indices_in, const Tensor& vertices_in,
                                                                              uintptr_t cam_address, bool want_host_info) {
  require_cuda(indices_in, "indices");
  require_cuda(vertices_in, "vertices");
  const RmCamera* cam = camera(cam_address);
  const at::Device dev = vertices_in.device();
  c10::cuda::CUDAGuard guard(dev);
  const Tensor indices = i32(indices_in), vertices = f32(vertices_in);
  const int64_t T = indices.size(0), V = vertices.size(0), G = (int64_t)cam->grid_height * cam->grid_width;
  Tensor tiles_touched = empty({T}, at::kInt, dev), rect = empty({T, 4}, at::kInt, dev);
  Tensor vs_tetra = empty({T, 3}, at::kFloat, dev), circumcenter = empty({T, 3}, at::kFloat, dev);
  Tensor tile_ranges = empty({G, 2}, at::kInt, dev), visible = empty({T}, at::kBool, dev);
  const int64_t bytes = (int64_t)lib.rm_bin_workspace_bytes(T, G);
  Tensor info = empty({3}, at::kLong, dev), workspace = empty({bytes}, at::kByte, dev);
  std::unique_ptr<PendingInfo> pending;
  if (want_host_info) pending = std::make_unique<PendingInfo>(c10::cuda::getCurrentCUDAStream(dev.index()));
  check(lib.rm_project_and_bin_visible(ptr<int32_t>(indices), T, ptr<float>(vertices), V, cam, ptr<int32_t>(tiles_touched),
                                       ptr<int32_t>(rect), ptr<float>(vs_tetra), ptr<float>(circumcenter),
                                       ptr<int32_t>(tile_ranges), ptr<RmBinInfo>(info), workspace.data_ptr(), bytes,
                                       ptr<uint8_t>(visible), pending ? ptr<RmBinInfo>(pending->block) : nullptr,
                                       stream_of(vertices)));
  if (pending) pending->record();
  std::vector<Tensor> out = {indices, vertices, tiles_touched, rect, vs_tetra, circumcenter, tile_ranges, info, workspace,
                             visible};
  return {std::move(out), std::move(pending)};
}

Tensor build_tile_lists(const Tensor& rect, const Tensor& tile_ranges, const Tensor& workspace, uintptr_t cam_address,
                        int64_t n_keys, int64_t n_region_keys) {
  const RmCamera* cam = camera(cam_address);
  const at::Device dev = rect.device();
  c10::cuda::CUDAGuard guard(dev);
  Tensor list = empty({n_keys}, at::kInt, dev);
  if (n_keys == 0) return list;
  const int64_t bytes = (int64_t)lib.rm_list_scratch_bytes(n_region_keys, cam->grid_height, cam->grid_width);
  if (bytes == 0) throw std::runtime_error("rm_b200: tile grids above 2^22 regions of 8 x 4 tiles are not supported");
  Tensor scratch = empty({bytes}, at::kByte, dev);
  check(lib.rm_build_tile_lists(ptr<int32_t>(rect), ptr<int32_t>(tile_ranges), rect.size(0), cam, n_keys, n_region_keys,
                                workspace.data_ptr(), scratch.data_ptr(), bytes, ptr<int32_t>(list), stream_of(rect)));
  return list;
}

Tensor pack_records(const Tensor& indices_in, const Tensor& vertices_in, const Tensor& cell_in, uintptr_t cam_address,
                    const c10::optional<Tensor>& tiles_touched, const c10::optional<Tensor>& clear_a,
                    const c10::optional<Tensor>& clear_b) {
  const at::Device dev = vertices_in.device();
  c10::cuda::CUDAGuard guard(dev);
  const Tensor indices = i32(indices_in), vertices = f32(vertices_in), cell = f32(cell_in);
  const int64_t T = indices.size(0);
  Tensor records = empty({T, RM_RECORD_FLOATS}, at::kFloat, dev);
  check(lib.rm_pack_records_and_clear(ptr<int32_t>(indices), ptr<float>(vertices), ptr<float>(cell), T, vertices.size(0),
                                      camera(cam_address), ptr<int32_t>(tiles_touched), ptr<float>(records),
                                      ptr<uint8_t>(clear_a), ptr<uint8_t>(clear_b), stream_of(vertices)));
  return records;
}

// Forward integration.  Returns (output_img, distortion_img, n_contributors) and, if `tet_flags` (zero-filled) is given,
// the hit lists' counts, ids and masks.
std::vector<Tensor> forward(const Tensor& list, const Tensor& tile_ranges, const Tensor& records, uintptr_t cam_address,
                            bool zero_fill, const c10::optional<Tensor>& jitter, const c10::optional<Tensor>& tet_flags) {
  const RmCamera* cam = camera(cam_address);
  const at::Device dev = records.device();
  c10::cuda::CUDAGuard guard(dev);
  const int64_t H = cam->image_height, W = cam->image_width;
  auto alloc = [&](at::IntArrayRef size, at::ScalarType type) {
    const auto o = at::TensorOptions().dtype(type).device(dev);
    return zero_fill ? at::zeros(size, o) : at::empty(size, o);
  };
  std::vector<Tensor> out = {alloc({H, W, 4}, at::kFloat), alloc({H, W, 5}, at::kFloat), alloc({H, W, 1}, at::kInt)};
  RmHitList hits = {nullptr, nullptr, nullptr, nullptr};
  if (tet_flags.has_value()) {
    const int64_t groups = ((int64_t)cam->tile_width * cam->tile_height + 15) / 16;
    const int64_t slots = std::max<int64_t>(list.size(0) * groups, 1);
    const int64_t units = (int64_t)cam->grid_height * cam->grid_width * groups;
    out.push_back(alloc({units}, at::kInt));
    out.push_back(empty({slots}, at::kInt, dev));
    out.push_back(empty({slots + 16 * units}, at::kShort, dev));
    hits = {ptr<int32_t>(out[3]), ptr<int32_t>(out[4]), ptr<uint16_t>(out[5]), ptr<uint8_t>(tet_flags)};
  }
  const bool any = tet_flags.has_value();
  extents({{kList, list.size(0)}, {kTets, records.size(0)}, {kHitIds, any ? out[4].size(0) : 0},
           {kHitMasks, any ? out[5].size(0) : 0}, {kUnits, any ? out[3].size(0) : 0}});
  check(lib.rm_forward_sized(ptr<int32_t>(list), ptr<int32_t>(tile_ranges), ptr<float>(records), cam, ptr<float>(jitter),
                             ptr<float>(out[0]), ptr<float>(out[1]), ptr<int32_t>(out[2]), any ? &hits : nullptr,
                             list.size(0), stream_of(records)));
  return out;
}

// What blend_forward does before its walk; tet_flags if need_grad.
struct Packed {
  Tensor tet_alive, indices, vertices, cell, records;
  c10::optional<Tensor> tet_flags;
};
Packed pack_for_blend(const Tensor& indices_in, const Tensor& vertices_in, const Tensor& cell_in, uintptr_t cam_address,
                                   const c10::optional<Tensor>& tiles_touched, bool need_grad) {
  require_cuda(vertices_in, "vertices");
  const at::Device dev = vertices_in.device();
  c10::cuda::CUDAGuard guard(dev);
  const Tensor indices = i32(indices_in), vertices = f32(vertices_in), cell = f32(cell_in);
  const int64_t T = indices.size(0);
  // tet_alive is never written by the reference kernel either: always False
  Tensor tet_alive = empty({T}, at::kBool, dev);
  c10::optional<Tensor> flags;
  if (need_grad) flags = empty({std::max<int64_t>(T, 1)}, at::kByte, dev);
  Tensor records = pack_records(indices, vertices, cell, cam_address, tiles_touched, tet_alive, flags);
  return {tet_alive, indices, vertices, cell, records, flags};
}

// The same ahead of a blend of these arguments; nothing where they are not such as it takes.
std::unique_ptr<Packed> pack_ahead(const Tensor& indices, const Tensor& vertices, const Tensor& cell, uintptr_t cam_address,
                                   const Tensor& tiles_touched) {
  if (!cell.is_cuda() || cell.device() != vertices.device() || cell.dim() != 2 || cell.size(0) != indices.size(0) ||
      cell.size(1) != 7)
    return nullptr;
  return std::make_unique<Packed>(pack_for_blend(indices, vertices, cell, cam_address, tiles_touched,
                                                 vertices.requires_grad() || cell.requires_grad()));
}

// Everything AlphaBlendTiledRender.forward does.  Returns (output_img, distortion_img, tet_alive, indices, vertices, cell,
// records, n_contributors, tet_flags[, counts, ids, masks]); the bracketed ones if need_grad.  packed: what pack_ahead has
// returned for the same arguments.
std::vector<Tensor> blend_forward(const Tensor& list, const Tensor& tile_ranges, const Tensor& indices_in,
                                  const Tensor& vertices_in, const Tensor& cell_in, uintptr_t cam_address, bool zero_fill,
                                  const c10::optional<Tensor>& jitter_in, const c10::optional<Tensor>& tiles_touched,
                                  bool need_grad, const Packed* packed) {
  const Packed p =
      packed ? *packed : pack_for_blend(indices_in, vertices_in, cell_in, cam_address, tiles_touched, need_grad);
  if (need_grad != p.tet_flags.has_value()) throw std::runtime_error("rm_b200: records packed for another kind of blend");
  c10::cuda::CUDAGuard guard(vertices_in.device());
  c10::optional<Tensor> jitter;
  if (jitter_in.has_value()) jitter = f32(*jitter_in);
  std::vector<Tensor> f = forward(list, tile_ranges, p.records, cam_address, zero_fill, jitter, p.tet_flags);
  std::vector<Tensor> out = {f[0], f[1], p.tet_alive, p.indices, p.vertices, p.cell, p.records, f[2]};
  if (need_grad) {
    out.push_back(*p.tet_flags);
    out.insert(out.end(), f.begin() + 3, f.end());
  }
  return out;
}

// The backward integration: (vertices_grad, cell_values_grad), both in one allocation (the second one 16-byte aligned), so
// that a multi-GPU job can sum them over the ranks with a single all-reduce.
std::tuple<Tensor, Tensor> backward(const Tensor& list, const Tensor& tile_ranges, const Tensor& records,
                                    uintptr_t cam_address, const c10::optional<Tensor>& jitter, const Tensor& output_img,
                                    const Tensor& distortion_img, const Tensor& n_contributors, const Tensor& counts,
                                    const Tensor& ids, const Tensor& masks, const Tensor& tet_flags, const Tensor& g_img_in,
                                    const Tensor& g_dist_in, const Tensor& indices, const Tensor& vertices,
                                    const Tensor& cell) {
  const at::Device dev = records.device();
  c10::cuda::CUDAGuard guard(dev);
  const int64_t T = indices.size(0), V = vertices.size(0), off = (3 * V + 3) / 4 * 4;
  const Tensor g_img = f32(g_img_in), g_dist = f32(g_dist_in);
  Tensor grad_records = empty({T, RM_GRAD_RECORD_FLOATS}, at::kFloat, dev), flat = empty({off + 7 * T}, at::kFloat, dev);
  if (off > 3 * V) flat.slice(0, 3 * V, off).zero_();
  Tensor vertices_grad = flat.slice(0, 0, 3 * V).view({V, 3}), cell_grad = flat.slice(0, off).view({T, 7});
  const RmHitList hits = {ptr<int32_t>(counts), ptr<int32_t>(ids), ptr<uint16_t>(masks), ptr<uint8_t>(tet_flags)};
  extents({{kList, list.size(0)}, {kTets, T}, {kVerts, V}, {kHitIds, ids.size(0)}, {kHitMasks, masks.size(0)},
           {kUnits, counts.size(0)}});
  check(lib.rm_backward(ptr<int32_t>(list), ptr<int32_t>(tile_ranges), ptr<float>(records), camera(cam_address),
                        ptr<float>(jitter), ptr<float>(output_img), ptr<float>(distortion_img), ptr<int32_t>(n_contributors),
                        &hits, ptr<float>(g_img), ptr<float>(g_dist), ptr<int32_t>(indices), ptr<float>(vertices),
                        ptr<float>(cell), T, V, ptr<float>(grad_records), ptr<float>(vertices_grad), ptr<float>(cell_grad),
                        stream_of(records)));
  return {vertices_grad, cell_grad};
}

Tensor distortion_loss(const Tensor& distortion_img) {
  const at::Device dev = distortion_img.device();
  c10::cuda::CUDAGuard guard(dev);
  const Tensor d = f32(distortion_img);
  Tensor partials = empty({RM_LOSS_PARTIALS}, at::kFloat, dev), loss = empty({}, at::kFloat, dev);
  check(lib.rm_distortion_loss(ptr<float>(d), d.numel() / 5, ptr<float>(partials), ptr<float>(loss), stream_of(d)));
  return loss;
}

Tensor distortion_loss_backward(const Tensor& distortion_img, const Tensor& grad_loss) {
  const at::Device dev = distortion_img.device();
  c10::cuda::CUDAGuard guard(dev);
  const Tensor d = f32(distortion_img), g = f32(grad_loss);
  Tensor out = at::empty_like(d);
  check(lib.rm_distortion_loss_backward(ptr<float>(d), d.numel() / 5, ptr<float>(g), ptr<float>(out), stream_of(d)));
  return out;
}

}  // namespace

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
  py::class_<Camera>(m, "Camera")
      .def(py::init<const py::object&, const at::Device&, const py::object&>())
      .def_property_readonly("address", [](const Camera& c) { return reinterpret_cast<uintptr_t>(&c.c); })
      .def_property_readonly("band_rows_only", [](const Camera& c) { return c.band_rows_only; })
      .def_property_readonly("grid", [](const Camera& c) { return std::make_tuple(c.c.grid_height, c.c.grid_width); })
      .def_property_readonly("zero_fill", [](const Camera& c) {
        return !(c.c.tile_row_begin == 0 && c.c.tile_row_end == c.c.grid_height) && !c.band_rows_only;
      });
  m.def("bind", &bind);
  // The interpreter lock is not held while a frame's memory is allocated and its kernels are launched (a launch waits when the
  // GPU's queue is full): other threads of the program, those of other GPUs among them, go on.
  py::call_guard<py::gil_scoped_release> unlocked;
  py::class_<PendingInfo>(m, "PendingInfo").def("wait", &PendingInfo::wait, unlocked);
  m.def("project_and_bin", &project_and_bin, unlocked);
  m.def("build_tile_lists", &build_tile_lists, unlocked);
  m.def("pack_records", &pack_records, unlocked);
  m.def("forward", &forward, unlocked);
  py::class_<Packed>(m, "Packed");
  m.def("pack_ahead", &pack_ahead, unlocked);
  m.def("blend_forward", &blend_forward, unlocked);
  m.def("blend_forward", [](const Tensor& list, const Tensor& tile_ranges, const Tensor& indices, const Tensor& vertices,
                            const Tensor& cell, uintptr_t cam, bool zero_fill, const c10::optional<Tensor>& jitter,
                            const c10::optional<Tensor>& tiles_touched, bool need_grad) {
    return blend_forward(list, tile_ranges, indices, vertices, cell, cam, zero_fill, jitter, tiles_touched, need_grad, nullptr);
  }, unlocked);
  m.def("backward", &backward, unlocked);
  m.def("distortion_loss", &distortion_loss, unlocked);
  m.def("distortion_loss_backward", &distortion_loss_backward, unlocked);
}
