// Host side of the operators: output allocation, argument checks, stream handling and the launches of the C ABI
// (include/sphconv_b200.h) in one native call per operator.
//
// An operator of this path is a handful of launches of a few microseconds each; driven from Python (one ctypes call and one
// torch.empty at a time, ~100 us a layer) a scan waited for the host, not for the GPU.  The library itself stays free of
// torch: this module loads it and calls it through the same entry points as any other binding.
#include <ATen/cuda/CUDAContext.h>
#include <ATen/cuda/CUDAEvent.h>
#include <c10/cuda/CUDACachingAllocator.h>
#include <c10/cuda/CUDAGuard.h>
#include <dlfcn.h>
#include <torch/extension.h>

#include <array>
#include <mutex>
#include <stdexcept>
#include <string>

#include "sphconv_b200.h"

namespace {

namespace py = pybind11;
using at::Tensor;
using std::optional;
using Ints = std::vector<int64_t>;

// ---- the C ABI -----------------------------------------------------------------------------------------------------
#define SPH_ENTRY_POINTS(X)                                                                                          \
  X(sph_last_error) X(sph_num_tiles) X(sph_tile_n_max) X(sph_rules_subm_scratch_bytes) X(sph_rules_subm)             \
  X(sph_rules_strided_scratch_bytes) X(sph_rules_strided_count_async) X(sph_rules_strided_fill) X(sph_rule_lists)    \
  X(sph_rules_to_nbr) X(sph_packed_weight_bytes) X(sph_pack_weight) X(sph_conv_gather) X(sph_conv_wgrad)             \
  X(sph_init_tensor_scratch_bytes) X(sph_init_tensor) X(sph_permute_rows) X(sph_dense_channels_first)                \
  X(sph_epilogue_backward) X(sph_voxel_transform) X(sph_voxel_feature_count) X(sph_voxelize_scratch_bytes)           \
  X(sph_voxelize_count) X(sph_voxelize_fill)

struct Abi {
#define X(name) decltype(&name) name = nullptr;
  SPH_ENTRY_POINTS(X)
#undef X
} abi;

void load(const std::string& path) {
  void* h = dlopen(path.c_str(), RTLD_NOW | RTLD_LOCAL);
  if (!h) throw std::runtime_error(std::string("sphconv_b200: ") + dlerror());
#define X(name)                                                                                        \
  abi.name = reinterpret_cast<decltype(&name)>(dlsym(h, #name));                                       \
  if (!abi.name) throw std::runtime_error("sphconv_b200: " #name " is missing from " + path);
  SPH_ENTRY_POINTS(X)
#undef X
}

template <typename T>
T check(T rc) {
  if (rc < 0)
    throw std::runtime_error(std::string("sphconv_b200: ") + abi.sph_last_error() + " (code " + std::to_string(rc) + ")");
  return rc;
}

[[noreturn]] void fail(const std::string& what) { throw std::runtime_error(what); }

// ---- arguments -----------------------------------------------------------------------------------------------------
void require_cuda(const Tensor& t) {
  if (!t.is_cuda())
    fail("sphconv_b200 ops run on CUDA tensors only (got a " + c10::DeviceTypeName(t.device().type(), true) +
         " tensor); there is no CPU path");
  if (!t.is_contiguous()) fail("sphconv_b200 ops need contiguous tensors");
}
void require_cuda(const optional<Tensor>& t) {
  if (t) require_cuda(*t);
}

void* ptr(const Tensor& t) { return t.data_ptr(); }
void* ptr(const optional<Tensor>& t) { return t ? t->data_ptr() : nullptr; }
int32_t* ints(const Tensor& t) { return static_cast<int32_t*>(t.data_ptr()); }
int32_t* ints(const optional<Tensor>& t) { return t ? ints(*t) : nullptr; }

int dtype_code(const Tensor& t, const char* what) {
  switch (t.scalar_type()) {
    case at::kFloat: return SPH_F32;
    case at::kHalf: return SPH_F16;
    case at::kBFloat16: return SPH_BF16;
    case at::kChar: return SPH_I8;
    default: fail(std::string("unsupported ") + what + " dtype " + c10::toString(t.scalar_type()));
  }
}

cudaStream_t stream_of(const Tensor& t) { return at::cuda::getCurrentCUDAStream(t.device().index()).stream(); }

Tensor empty(at::IntArrayRef shape, at::ScalarType type, const Tensor& like) {
  return at::empty(shape, at::TensorOptions().dtype(type).device(like.device()));
}

sph_geom geometry(int64_t B, const Ints& in, const Ints& out, const Ints& k, const Ints& s, const Ints& p, const Ints& d,
                  const Ints& tile) {
  if (in.size() < 3 || out.size() < 3 || k.size() < 3 || s.size() < 3 || p.size() < 3 || d.size() < 3 || tile.size() < 2)
    fail("shapes, kernel size, stride, padding and dilation have three entries, the tile two");
  sph_geom g;
  g.B = (int32_t)B;
  for (int i = 0; i < 3; ++i) {
    g.in_shape[i] = (int32_t)in[i];
    g.out_shape[i] = (int32_t)out[i];
    g.ksize[i] = (int32_t)k[i];
    g.stride[i] = (int32_t)s[i];
    g.padding[i] = (int32_t)p[i];
    if (d[i] < 1) fail("dilation must be positive");
    g.dilation[i] = (int32_t)d[i];
  }
  g.tile[0] = (int32_t)tile[0];
  g.tile[1] = (int32_t)tile[1];
  return g;
}

void check_index(const Tensor& z_idx, const Tensor& z_ptr) {
  require_cuda(z_idx);
  require_cuda(z_ptr);
  if (z_idx.scalar_type() != at::kInt || z_ptr.scalar_type() != at::kInt) fail("z_idx and z_ptr must be int32");
}

// ---- per-device state ----------------------------------------------------------------------------------------------
// The int32 word the kernels OR error bits into.
std::mutex state_mutex;
std::array<Tensor, 64> status_words;

Tensor status_tensor(int device) {
  if (device < 0 || device >= (int)status_words.size()) fail("device ordinal not supported");
  std::lock_guard<std::mutex> lock(state_mutex);
  Tensor& t = status_words[device];
  if (!t.defined()) t = at::zeros({1}, at::TensorOptions().dtype(at::kInt).device(at::kCUDA, device));
  return t;
}
int32_t* status_of(const Tensor& t) {
  const int device = t.device().index();
  Tensor& s = status_words.at(device);
  return ints(s.defined() ? s : status_tensor(device));
}

// The stream pair lists are written on, beside the convolution that reads the table only.
c10::cuda::CUDAStream side_stream(int device) {
  static std::array<optional<c10::cuda::CUDAStream>, 64> streams;
  std::lock_guard<std::mutex> lock(state_mutex);
  auto& s = streams.at(device);
  if (!s) s = c10::cuda::getStreamFromPool(false, device);
  return *s;
}
