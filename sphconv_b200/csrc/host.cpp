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

#include <algorithm>
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
  X(sph_rules_strided_scratch_bytes) X(sph_rules_strided_count) X(sph_rules_strided_fill) X(sph_rule_lists)    \
  X(sph_rules_to_nbr) X(sph_packed_weight_bytes) X(sph_pack_weight) X(sph_conv_gather) X(sph_conv_wgrad)             \
  X(sph_init_tensor_scratch_bytes) X(sph_init_tensor) X(sph_permute_rows) X(sph_dense_channels_first)                \
  X(sph_epilogue_backward) X(sph_voxel_transform) X(sph_voxel_feature_count) X(sph_voxelize_scratch_bytes)           \
  X(sph_voxelize_count) X(sph_voxelize_fill)

struct Abi {
#define X(name) decltype(&::name) name = nullptr;
  SPH_ENTRY_POINTS(X)
#undef X
} abi;

void load(const std::string& path) {
  void* h = dlopen(path.c_str(), RTLD_NOW | RTLD_LOCAL);
  if (!h) throw std::runtime_error(std::string("sphconv_b200: ") + dlerror());
#define X(name)                                                                                        \
  abi.name = reinterpret_cast<decltype(&::name)>(dlsym(h, #name));                                       \
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
// The int32 word the kernels OR error bits into.  Looked up under the lock: autograd's threads come here without the GIL.
std::mutex state_mutex;
std::array<Tensor, 64> status_words;

Tensor status_tensor(int device) {
  if (device < 0 || device >= (int)status_words.size()) fail("device ordinal not supported");
  std::lock_guard<std::mutex> lock(state_mutex);
  Tensor& t = status_words[device];
  if (!t.defined()) {
    t = at::zeros({1}, at::TensorOptions().dtype(at::kInt).device(at::kCUDA, device));
    // kernels of other streams may be the next to write it
    if (c10::cuda::currentStreamCaptureStatusMayInitCtx() == c10::cuda::CaptureStatus::None)
      at::cuda::getCurrentCUDAStream(device).synchronize();
  }
  return t;
}
int32_t* status_of(const Tensor& t) { return ints(status_tensor(t.device().index())); }

// The stream pair lists are written on, beside the convolution that reads the table only.
c10::cuda::CUDAStream side_stream(int device) {
  static std::array<optional<c10::cuda::CUDAStream>, 64> streams;
  std::lock_guard<std::mutex> lock(state_mutex);
  auto& s = streams.at(device);
  if (!s) s = c10::cuda::getStreamFromPool(false, device);
  return *s;
}

// ---- rules ---------------------------------------------------------------------------------------------------------
// Marks the pair lists of a rule set complete: recorded on the side stream, joined once.
struct ListsReady {
  at::cuda::CUDAEvent event;
  void join() { event.block(at::cuda::getCurrentCUDAStream(event.device_index())); }
};

// The -1 padding of a rule set's lists, written on the side stream from the moment the lists are allocated: the fill is
// bound by HBM and the kernels that make the neighbour table by latency, so beside one another they cost little more than
// the longer of the two (a submanifold and a strided rule set with 207 MB of lists: 132 -> 118 us).  A fill below kBesideBytes takes
// about as long as the two events it would need and stays on the current stream, in front of the lists.
class Padding {
 public:
  static constexpr int64_t kBesideBytes = 16 << 20;
  Padding(const Tensor& rules, bool fill) {
    if (!fill || !rules.defined() || (int64_t)rules.nbytes() < kBesideBytes) return;
    const int device = rules.device().index();
    const auto side = side_stream(device);
    at::cuda::CUDAEvent allocated;
    allocated.record(at::cuda::getCurrentCUDAStream(device));
    allocated.block(side);
    C10_CUDA_CHECK(cudaMemsetAsync(rules.data_ptr(), 0xFF, rules.nbytes(), side));
    done_.record(side);
    device_ = device;
  }
  Padding(const Padding&) = delete;
  ~Padding() {                  // an error on the way: the lists are freed on the current stream, behind the fill
    if (begun()) try { join(); } catch (...) {}
  }
  bool begun() const { return device_ >= 0; }
  void join() {                 // the current stream continues behind the fill
    done_.block(at::cuda::getCurrentCUDAStream(device_));
    device_ = -1;
  }
  void leave() { device_ = -1; }   // the lists are written on the side stream too

 private:
  at::cuda::CUDAEvent done_;
  int device_ = -1;
};

// Rule sets from this size on have their lists written on the side stream where the caller asks for it, beside the convolution.  The two
// events, the waits and the allocator's records of a smaller one cost the host more than its lists cost the GPU (us, lists on the side /
// the caller's stream): one layer on 6 k rows 58 / 46, on 16 k 66 / 39, a strided layer's training step on 16 k to 71 k rows 228 / 206.
// From here on it is the layer that decides (lists_beside in sphconv_cuda.py).
constexpr int64_t kListsBesideRows = 100000;

// The lists of a rule set whose table has been enqueued on the current stream, on the side stream.
std::shared_ptr<ListsReady> lists_beside(const sph_geom& g, const Tensor& oz_ptr, const Tensor& nbr, int32_t tnm,
                                         const Tensor& rules, const Tensor& rule_size, bool fill) {
  const auto current = at::cuda::getCurrentCUDAStream(nbr.device().index());
  const auto side = side_stream(nbr.device().index());
  at::cuda::CUDAEvent table_done;
  table_done.record(current);
  table_done.block(side);
  check(abi.sph_rule_lists(ints(oz_ptr), &g, nbr.size(1), ints(nbr), tnm, ints(rules), ints(rule_size), fill,
                           status_of(nbr), side.stream()));
  auto ready = std::make_shared<ListsReady>();
  ready->event.record(side);
  for (const Tensor& t : {rules, rule_size, nbr, oz_ptr}) c10::cuda::CUDACachingAllocator::recordStream(t.storage().data_ptr(), side);
  return ready;
}

struct Lists {               // empty when the caller keeps the tables only
  Tensor rules, rule_size;
  int32_t tnm = 0;
};

Lists make_lists(const sph_geom& g, int64_t nnz, const Tensor& like, bool materialize) {
  Lists l;
  if (!materialize) return l;
  l.tnm = check(abi.sph_tile_n_max(&g, nnz));
  const int64_t kv = (int64_t)g.ksize[0] * g.ksize[1] * g.ksize[2], tiles = check(abi.sph_num_tiles(&g));
  l.rules = empty({tiles, kv, 2, l.tnm}, at::kInt, like);
  l.rule_size = empty({tiles, kv}, at::kInt, like);
  return l;
}

py::object or_none(const Tensor& t) { return t.defined() ? py::cast(t) : py::none(); }
py::object or_none(const std::shared_ptr<ListsReady>& r) { return r ? py::cast(r) : py::none(); }

// -> (rules, rule_size, nbr, ready)
py::tuple rules_subm(const Tensor& z_idx, const Tensor& z_ptr, int64_t B, const Ints& in, const Ints& out, const Ints& k,
                     const Ints& s, const Ints& p, const Ints& d, const Ints& tile, bool fill, bool materialize, bool defer) {
  check_index(z_idx, z_ptr);
  const c10::cuda::CUDAGuard guard(z_idx.device());
  const sph_geom g = geometry(B, in, out, k, s, p, d, tile);
  const int64_t nnz = z_idx.size(0), kv = k[0] * k[1] * k[2];
  Lists l = make_lists(g, nnz, z_idx, materialize);
  Padding padding(l.rules, fill && nnz > 0);
  defer = defer && materialize && nnz >= kListsBesideRows;
  Tensor nbr = empty({kv, nnz}, at::kInt, z_idx);
  const int64_t bytes = check(abi.sph_rules_subm_scratch_bytes(&g, nnz));
  Tensor scratch = bytes ? empty({bytes}, at::kByte, z_idx) : Tensor();
  const bool here = materialize && !defer && !padding.begun();
  check(abi.sph_rules_subm(ints(z_idx), ints(z_ptr), nnz, &g, bytes ? ptr(scratch) : nullptr, l.tnm,
                           here ? ints(l.rules) : nullptr, here ? ints(l.rule_size) : nullptr, ints(nbr), fill,
                           status_of(z_idx), stream_of(z_idx)));
  std::shared_ptr<ListsReady> ready;
  if (defer) {
    ready = lists_beside(g, z_ptr, nbr, l.tnm, l.rules, l.rule_size, fill && !padding.begun());
    padding.leave();
  } else if (padding.begun()) {
    padding.join();
    check(abi.sph_rule_lists(ints(z_ptr), &g, nnz, ints(nbr), l.tnm, ints(l.rules), ints(l.rule_size), false, status_of(nbr),
                             stream_of(nbr)));
  }
  return py::make_tuple(or_none(l.rules), or_none(l.rule_size), nbr, or_none(ready));
}

// Words of pinned host memory that kernels write row counts to, 1 KiB at a time; a word given back before the kernel that writes
// it has run waits for that kernel's event.  (An allocation of torch's pinned memory for every count took 2 us longer.)
class CountWords {
 public:
  int32_t* take() {
    std::lock_guard<std::mutex> lock(mutex_);
    if (free_.empty()) {
      auto done = std::partition(busy_.begin(), busy_.end(), [](const auto& b) { return !b.first.query(); });
      for (auto b = done; b != busy_.end(); ++b) free_.push_back(b->second);
      busy_.erase(done, busy_.end());
    }
    if (free_.empty()) {
      void* words = nullptr;
      C10_CUDA_CHECK(cudaHostAlloc(&words, kWords * sizeof(int32_t), cudaHostAllocMapped | cudaHostAllocPortable));
      for (int i = 0; i < kWords; ++i) free_.push_back(static_cast<int32_t*>(words) + i);
    }
    int32_t* word = free_.back();
    free_.pop_back();
    return word;
  }
  void give(int32_t* word) {
    std::lock_guard<std::mutex> lock(mutex_);
    free_.push_back(word);
  }
  void give(int32_t* word, at::cuda::CUDAEvent&& written) {
    std::lock_guard<std::mutex> lock(mutex_);
    busy_.emplace_back(std::move(written), word);
  }

 private:
  static constexpr int kWords = 256;
  std::mutex mutex_;
  std::vector<int32_t*> free_;
  std::vector<std::pair<at::cuda::CUDAEvent, int32_t*>> busy_;
};
CountWords& count_words() {
  static CountWords* words = new CountWords;      // outlives the interpreter's last handles
  return *words;
}

// Step 1 of a strided rule set, enqueued; the row count is in the word once the step has run.  The word is the handle's own: any
// number of them may be outstanding, for any time.
struct Pending {
  sph_geom g;
  Tensor z_idx, z_ptr, scratch, oz_ptr;
  c10::cuda::CUDAStream stream;
  at::cuda::CUDAEvent event;
  int32_t* word = count_words().take();
  bool enqueued = false, read = false;

  explicit Pending(c10::cuda::CUDAStream s) : stream(s) {}
  Pending(const Pending&) = delete;
  ~Pending() {
    try {
      if (!enqueued || read) count_words().give(word);
      else count_words().give(word, std::move(event));
    } catch (...) {                 // the word is lost
    }
  }
  int64_t count() {
    event.synchronize();
    read = true;
    return *const_cast<const volatile int32_t*>(word);
  }

  bool matches(const Tensor& zi, const Tensor& zp, const sph_geom& o) const {
    return zi.is_same(z_idx) && zp.is_same(z_ptr) && std::memcmp(&g, &o, sizeof(g)) == 0;
  }
};

std::shared_ptr<Pending> strided_begin(const Tensor& z_idx, const Tensor& z_ptr, int64_t B, const Ints& in, const Ints& out,
                                       const Ints& k, const Ints& s, const Ints& p, const Ints& d, const Ints& tile) {
  check_index(z_idx, z_ptr);
  const c10::cuda::CUDAGuard guard(z_idx.device());
  auto r = std::make_shared<Pending>(at::cuda::getCurrentCUDAStream(z_idx.device().index()));
  r->g = geometry(B, in, out, k, s, p, d, tile);
  r->z_idx = z_idx;
  r->z_ptr = z_ptr;
  const int64_t nnz = z_idx.size(0);
  r->scratch = empty({check(abi.sph_rules_strided_scratch_bytes(&r->g, nnz))}, at::kByte, z_idx);
  r->oz_ptr = empty({B, out[0], out[1]}, at::kInt, z_idx);
  check(abi.sph_rules_strided_count(ints(z_idx), ints(z_ptr), nnz, &r->g, ptr(r->scratch), ints(r->oz_ptr), r->word, nullptr,
                                    r->stream.stream()));
  r->event.record(r->stream);
  r->enqueued = true;
  return r;
}

// -> (oz_idx, oz_ptr, rules, rule_size, nbr, nbr_t, ready)
py::tuple strided_rules(const Tensor& z_idx, const Tensor& z_ptr, int64_t B, const Ints& in, const Ints& out, const Ints& k,
                        const Ints& s, const Ints& p, const Ints& d, const Ints& tile, std::shared_ptr<Pending> pending,
                        bool fill, bool materialize, bool transposed, bool defer) {
  const sph_geom g = geometry(B, in, out, k, s, p, d, tile);
  if (!pending || !pending->matches(z_idx, z_ptr, g)) pending = strided_begin(z_idx, z_ptr, B, in, out, k, s, p, d, tile);
  const c10::cuda::CUDAGuard guard(z_idx.device());
  const auto current = at::cuda::getCurrentCUDAStream(z_idx.device().index());
  if (current != pending->stream)        // begun on another stream, whose allocator must not reuse them under this one's kernels
    for (const Tensor& t : {pending->scratch, pending->oz_ptr})
      c10::cuda::CUDACachingAllocator::recordStream(t.storage().data_ptr(), current);
  const int64_t nnz = z_idx.size(0), kv = k[0] * k[1] * k[2];
  // everything that does not need the row count is made before the wait for it
  Lists l = make_lists(g, nnz, z_idx, materialize);
  Padding padding(l.rules, fill);
  Tensor nbr_t = transposed ? empty({kv, nnz}, at::kInt, z_idx) : Tensor();
  int64_t n_out;
  {
    py::gil_scoped_release release;
    n_out = pending->count();
  }
  defer = defer && materialize && n_out >= kListsBesideRows;
  Tensor oz_idx = empty({n_out}, at::kInt, z_idx);
  Tensor nbr = empty({kv, n_out}, at::kInt, z_idx);
  const bool here = materialize && !defer && !padding.begun();
  check(abi.sph_rules_strided_fill(ints(z_idx), ints(z_ptr), nnz, &g, ptr(pending->scratch), ints(pending->oz_ptr), n_out,
                                   l.tnm, ints(oz_idx), here ? ints(l.rules) : nullptr, here ? ints(l.rule_size) : nullptr,
                                   ints(nbr), transposed ? ints(nbr_t) : nullptr, fill, status_of(z_idx), stream_of(z_idx)));
  std::shared_ptr<ListsReady> ready;
  if (defer) {
    ready = lists_beside(g, pending->oz_ptr, nbr, l.tnm, l.rules, l.rule_size, fill && !padding.begun());
    padding.leave();
  } else if (padding.begun()) {
    padding.join();
    check(abi.sph_rule_lists(ints(pending->oz_ptr), &g, n_out, ints(nbr), l.tnm, ints(l.rules), ints(l.rule_size), false,
                             status_of(nbr), stream_of(nbr)));
  }
  return py::make_tuple(oz_idx, pending->oz_ptr, or_none(l.rules), or_none(l.rule_size), nbr, or_none(nbr_t), or_none(ready));
}

// The lists of a finished table as a step of its own (the caller times it), on the side stream or the current one.
// -> (rules, rule_size, ready)
py::tuple lists_of_table(const Tensor& oz_ptr, const Tensor& nbr, int64_t nnz, int64_t B, const Ints& in, const Ints& out,
                         const Ints& k, const Ints& s, const Ints& p, const Ints& d, const Ints& tile, bool fill, bool beside) {
  const c10::cuda::CUDAGuard guard(nbr.device());
  const sph_geom g = geometry(B, in, out, k, s, p, d, tile);
  const Lists l = make_lists(g, nnz, nbr, true);
  std::shared_ptr<ListsReady> ready;
  if (beside) ready = lists_beside(g, oz_ptr, nbr, l.tnm, l.rules, l.rule_size, fill);
  else
    check(abi.sph_rule_lists(ints(oz_ptr), &g, nbr.size(1), ints(nbr), l.tnm, ints(l.rules), ints(l.rule_size), fill,
                             status_of(nbr), stream_of(nbr)));
  return py::make_tuple(l.rules, l.rule_size, or_none(ready));
}

// rules / rule_size with a capacity of exactly the longest list: count, read the maximum, allocate, fill.
py::tuple exact_lists(const Tensor& oz_ptr, const Tensor& nbr, int64_t B, const Ints& in, const Ints& out, const Ints& k,
                      const Ints& s, const Ints& p, const Ints& d, const Ints& tile, bool fill) {
  const c10::cuda::CUDAGuard guard(nbr.device());
  const sph_geom g = geometry(B, in, out, k, s, p, d, tile);
  const int64_t tiles = check(abi.sph_num_tiles(&g)), kv = nbr.size(0);
  Tensor rule_size = empty({tiles, kv}, at::kInt, nbr);
  check(abi.sph_rule_lists(ints(oz_ptr), &g, nbr.size(1), ints(nbr), 0, nullptr, ints(rule_size), 0, status_of(nbr), stream_of(nbr)));
  const int64_t tnm = rule_size.numel() ? std::max<int64_t>(1, rule_size.max().item<int64_t>()) : 1;
  Tensor rules = empty({tiles, kv, 2, tnm}, at::kInt, nbr);
  check(abi.sph_rule_lists(ints(oz_ptr), &g, nbr.size(1), ints(nbr), (int32_t)tnm, ints(rules), ints(rule_size), fill,
                           status_of(nbr), stream_of(nbr)));
  return py::make_tuple(rules, rule_size);
}

// Tables of a reference-format rules tensor made elsewhere.  -> (nbr, nbr_t)
py::tuple rules_to_nbr(const Tensor& rules, const Tensor& rule_size, int64_t n_in, int64_t n_out, bool want_nbr, bool want_t) {
  require_cuda(rules);
  require_cuda(rule_size);
  const c10::cuda::CUDAGuard guard(rules.device());
  const int64_t kv = rules.size(1);
  Tensor nbr = want_nbr ? empty({kv, n_out}, at::kInt, rules) : Tensor();
  Tensor nbr_t = want_t ? empty({kv, n_in}, at::kInt, rules) : Tensor();
  check(abi.sph_rules_to_nbr(ints(rules), ints(rule_size), (int32_t)rules.size(0), (int32_t)kv, (int32_t)rules.size(3), n_in,
                             n_out, want_nbr ? ints(nbr) : nullptr, want_t ? ints(nbr_t) : nullptr, status_of(rules),
                             stream_of(rules)));
  return py::make_tuple(or_none(nbr), or_none(nbr_t));
}

// ---- convolution ---------------------------------------------------------------------------------------------------
// UMMA image of a [KV, K, N] weight, or None where a CUDA-core kernel runs.
optional<Tensor> pack_weight(const Tensor& w) {
  require_cuda(w);             // the image is made from the raw memory: of an expanded weight that is too short
  const int code = dtype_code(w, "weight");
  const int32_t kv = (int32_t)w.size(0), k = (int32_t)w.size(1), n = (int32_t)w.size(2);
  const int64_t bytes = abi.sph_packed_weight_bytes(code, kv, k, n);
  if (bytes <= 0) return std::nullopt;
  const c10::cuda::CUDAGuard guard(w.device());
  Tensor packed = empty({bytes}, at::kByte, w);
  check(abi.sph_pack_weight(ptr(w), code, kv, k, n, ptr(packed), stream_of(w)));
  return packed;
}

Tensor conv_gather(const Tensor& rows, const Tensor& weight, const optional<Tensor>& packed, const Tensor& nbr, int64_t n_out,
                   bool flip, const optional<Tensor>& scale, const optional<Tensor>& bias, bool relu,
                   optional<at::ScalarType> out_dtype) {
  require_cuda(rows);
  require_cuda(weight);
  require_cuda(nbr);
  require_cuda(scale);
  require_cuda(bias);
  const int code = dtype_code(rows, "feature");
  if (weight.scalar_type() != rows.scalar_type())
    fail(std::string("feature (") + c10::toString(rows.scalar_type()) + ") and weight (" + c10::toString(weight.scalar_type()) +
         ") dtypes differ");
  const int64_t kv = weight.size(0), k_ch = weight.size(1), n_ch = weight.size(2);
  if (rows.dim() != 2 || rows.size(1) != k_ch)
    fail("feature has " + std::to_string(rows.size(-1)) + " channels, weight expects " + std::to_string(k_ch));
  const bool bias_16 = bias && rows.itemsize() == 2 && bias->scalar_type() == rows.scalar_type();
  for (const auto* v : {&scale, &bias})
    if (*v && (((*v)->scalar_type() != at::kFloat && !(v == &bias && bias_16)) || (*v)->numel() != n_ch))
      fail("scale / bias must be float32 [out_channels] (the bias may have the features' 16-bit type)");
  Tensor out = empty({n_out, n_ch}, out_dtype.value_or(code == SPH_I8 ? at::kFloat : rows.scalar_type()), rows);
  if (n_out == 0) return out;
  const c10::cuda::CUDAGuard guard(rows.device());
  check(abi.sph_conv_gather(ptr(rows), code, rows.size(0), ptr(weight), ptr(packed), ints(nbr), n_out, (int32_t)kv,
                            (int32_t)k_ch, (int32_t)n_ch, flip, static_cast<const float*>(ptr(scale)), ptr(bias),
                            (relu ? 1 : 0) | (bias_16 ? SPH_BIAS_IN_ROW_TYPE : 0), ptr(out), dtype_code(out, "output"),
                            status_of(rows), stream_of(rows)));
  return out;
}

Tensor conv_wgrad(const Tensor& feature, const Tensor& d_out, const Tensor& nbr, const optional<Tensor>& out, bool accumulate) {
  require_cuda(feature);
  require_cuda(d_out);
  require_cuda(out);
  if (feature.scalar_type() != d_out.scalar_type()) fail("feature and gradient dtypes differ");
  const int64_t kv = nbr.size(0), k_ch = feature.size(1), n_ch = d_out.size(1);
  if (out && (out->scalar_type() != at::kFloat || out->numel() != kv * k_ch * n_ch))
    fail("out must be float32 with " + std::to_string(kv) + " x " + std::to_string(k_ch) + " x " + std::to_string(n_ch) + " elements");
  const c10::cuda::CUDAGuard guard(feature.device());
  Tensor dw = out ? *out : empty({kv, k_ch, n_ch}, at::kFloat, feature);
  check(abi.sph_conv_wgrad(ptr(feature), ptr(d_out), dtype_code(feature, "feature"), feature.size(0), ints(nbr), d_out.size(0),
                           (int32_t)kv, (int32_t)k_ch, (int32_t)n_ch, static_cast<float*>(ptr(dw)), out && accumulate ? 0 : 1,
                           status_of(feature), stream_of(feature)));
  return dw;
}

std::pair<Tensor, Tensor> epilogue_grads(const Tensor& d_out, const optional<Tensor>& out, bool relu, bool need_bias) {
  require_cuda(d_out);
  require_cuda(out);
  const int64_t n = d_out.size(0), ch = d_out.size(1);
  if (d_out.scalar_type() == at::kChar || ch > 256)
    fail("epilogue_backward: float32 / float16 / bfloat16 gradients with at most 256 channels");
  const c10::cuda::CUDAGuard guard(d_out.device());
  Tensor d_pre = relu ? at::empty_like(d_out) : Tensor();
  Tensor d_bias = need_bias ? empty({ch}, at::kFloat, d_out) : Tensor();
  if (relu || need_bias)
    check(abi.sph_epilogue_backward(ptr(d_out), relu ? ptr(out) : nullptr, dtype_code(d_out, "gradient"), n, (int32_t)ch, relu,
                                    relu ? ptr(d_pre) : nullptr, need_bias ? static_cast<float*>(ptr(d_bias)) : nullptr,
                                    stream_of(d_out)));
  return {d_pre, d_bias};
}

// -> (d_pre or None, d_bias or None)
py::tuple epilogue_backward(const Tensor& d_out, const optional<Tensor>& out, bool relu, bool need_bias) {
  const auto r = epilogue_grads(d_out, out, relu, need_bias);
  return py::make_tuple(or_none(r.first), or_none(r.second));
}

// The differentiable layer: relu(conv + bias) with its gradients, as sphconv_b200.functional.ConvFunction computes them (the
// reference's sphconv/functional.py:12-78), without a trip through Python in either direction.
struct ConvLayer : public torch::autograd::Function<ConvLayer> {
  static Tensor forward(torch::autograd::AutogradContext* ctx, const Tensor& feature, const Tensor& weight,
                        const optional<Tensor>& bias, const Tensor& nbr, const optional<Tensor>& nbr_t, int64_t n_out, bool relu) {
    at::AutoDispatchBelowADInplaceOrView guard;
    optional<Tensor> b;                  // float32, or the features' 16-bit type as it is
    if (bias) b = (feature.itemsize() == 2 && bias->scalar_type() == feature.scalar_type() ? bias->detach() : bias->detach().to(at::kFloat)).contiguous();
    Tensor out = conv_gather(feature, weight, pack_weight(weight), nbr, n_out, false, std::nullopt, b, relu, std::nullopt);
    ctx->save_for_backward({feature, weight, relu ? out : Tensor(), nbr, nbr_t.value_or(Tensor())});
    ctx->saved_data["relu"] = relu;
    ctx->saved_data["bias"] = bias ? (int64_t)bias->scalar_type() : (int64_t)-1;
    return out;
  }

  static torch::autograd::variable_list backward(torch::autograd::AutogradContext* ctx, torch::autograd::variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    const Tensor &feature = saved[0], &weight = saved[1], &out = saved[2], &nbr = saved[3], &nbr_t = saved[4];
    const bool relu = ctx->saved_data["relu"].toBool();
    const int64_t bias_type = ctx->saved_data["bias"].toInt();
    Tensor d_out = grads[0].contiguous(), d_feature, d_weight, d_bias;
    const c10::cuda::CUDAGuard guard(d_out.device());
    if (relu || bias_type >= 0) {        // gradient mask and bias gradient in one pass over the rows
      auto r = epilogue_grads(d_out, relu ? optional<Tensor>(out) : std::nullopt, relu, bias_type >= 0);
      if (relu) d_out = r.first;
      if (bias_type >= 0) d_bias = r.second.to((at::ScalarType)bias_type);
    }
    if (ctx->needs_input_grad(0)) {
      // the transposed table, or - (i,o) at k is (o,i) at KV-1-k in an odd-kernel submanifold layer - the forward one, flipped
      const Tensor wt = weight.transpose(1, 2).contiguous();
      d_feature = conv_gather(d_out, wt, pack_weight(wt), nbr_t.defined() ? nbr_t : nbr, feature.size(0), !nbr_t.defined(),
                              std::nullopt, std::nullopt, false, std::nullopt);
    }
    if (ctx->needs_input_grad(1)) d_weight = conv_wgrad(feature, d_out, nbr, std::nullopt, false).to(feature.scalar_type());
    return {d_feature, d_weight, d_bias, Tensor(), Tensor(), Tensor(), Tensor()};
  }
};

Tensor conv_layer(const Tensor& feature, const Tensor& weight, const optional<Tensor>& bias, const Tensor& nbr,
                  const optional<Tensor>& nbr_t, int64_t n_out, bool relu) {
  return ConvLayer::apply(feature, weight, bias, nbr, nbr_t, n_out, relu);
}

// ---- tensor operations ---------------------------------------------------------------------------------------------
// COO rows -> (rows in range-voxel order, z_idx, z_ptr, permutation)
py::tuple init_tensor(const Tensor& feature_in, const Tensor& indices, int64_t B, const Ints& shape) {
  require_cuda(feature_in);
  require_cuda(indices);
  if (indices.dim() != 2 || indices.size(1) != 4 || indices.is_floating_point()) fail("indices must be an integer tensor [NNZ, 4]");
  if (feature_in.dim() != 2 || feature_in.size(0) != indices.size(0)) fail("feature must be [NNZ, C] with one row per index");
  const c10::cuda::CUDAGuard guard(feature_in.device());
  const Tensor feature = feature_in.contiguous();
  const Tensor idx = indices.to(at::kInt).contiguous();
  const int64_t nnz = feature.size(0);
  const int32_t dims[3] = {(int32_t)shape.at(0), (int32_t)shape.at(1), (int32_t)shape.at(2)};
  Tensor out = at::empty_like(feature);
  Tensor z_idx = empty({nnz}, at::kInt, feature), perm = empty({nnz}, at::kInt, feature);
  Tensor z_ptr = empty({B, shape[0], shape[1]}, at::kInt, feature);
  Tensor scratch = empty({check(abi.sph_init_tensor_scratch_bytes((int32_t)B, dims))}, at::kByte, feature);
  check(abi.sph_init_tensor(ptr(feature), (int32_t)(feature.size(1) * feature.element_size()), nnz, ints(idx), (int32_t)B, dims,
                            ptr(scratch), ptr(out), ints(z_idx), ints(z_ptr), ints(perm), status_of(feature), stream_of(feature)));
  return py::make_tuple(out, z_idx, z_ptr, perm);
}

// out[n] = rows[permutation[n]]
Tensor gather_rows(const Tensor& rows_in, const Tensor& permutation) {
  require_cuda(rows_in);
  require_cuda(permutation);
  if (permutation.scalar_type() != at::kInt) fail("permutation must be int32");
  const c10::cuda::CUDAGuard guard(rows_in.device());
  const Tensor rows = rows_in.contiguous();
  Tensor out = at::empty_like(rows);
  check(abi.sph_permute_rows(ptr(rows), (int32_t)(rows.size(1) * rows.element_size()), rows.size(0), ints(permutation), 1,
                             ptr(out), stream_of(rows)));
  return out;
}

// rows [NNZ,C] <-> dense [B,C,s0,s1,s2]
Tensor dense_channels_first(const Tensor& from, const Tensor& z_idx, const Tensor& z_ptr, const Ints& shape, bool backward) {
  require_cuda(from);
  require_cuda(z_idx);
  require_cuda(z_ptr);
  const c10::cuda::CUDAGuard guard(from.device());
  const int64_t nnz = backward ? z_idx.size(0) : std::min(from.size(0), z_idx.size(0));
  const int32_t dims[3] = {(int32_t)shape.at(2), (int32_t)shape.at(3), (int32_t)shape.at(4)};
  Tensor out = backward ? empty({nnz, shape[1]}, from.scalar_type(), from) : empty(shape, from.scalar_type(), from);
  const Tensor& rows = backward ? out : from;
  const Tensor& dense = backward ? from : out;
  check(abi.sph_dense_channels_first(ptr(rows), (int32_t)from.element_size(), (int32_t)shape[1], nnz, ints(z_idx), ints(z_ptr),
                                     (int32_t)shape[0], dims, ptr(dense), backward, status_of(from), stream_of(from)));
  return out;
}

// ---- voxeliser -----------------------------------------------------------------------------------------------------
Tensor voxel_transform(const Tensor& points, int64_t system) {
  require_cuda(points);
  if (points.scalar_type() != at::kFloat || points.dim() != 2 || points.size(1) < 4)
    fail("points must be a float32 tensor [N, >=4]");
  const c10::cuda::CUDAGuard guard(points.device());
  Tensor sys = empty({points.size(0), 4}, at::kFloat, points);
  check(abi.sph_voxel_transform(static_cast<const float*>(ptr(points)), (int32_t)points.size(1), points.size(0), (int)system,
                                static_cast<float*>(ptr(sys)), stream_of(points)));
  return sys;
}

// -> (feature, z_idx, z_ptr, coordinates, number of points)
py::tuple voxelize(const Tensor& points, const optional<Tensor>& scan_ptr, const Tensor& sys, const Ints& cells,
                   const std::vector<double>& range, int64_t max_points, int64_t max_voxels, int64_t append_mode,
                   bool with_coordinates) {
  require_cuda(points);
  require_cuda(sys);
  const int64_t n = points.size(0);
  if (sys.scalar_type() != at::kFloat || sys.dim() != 2 || sys.size(0) != n || sys.size(1) != 4)
    fail("system_points must be float32 [N, 4]");
  const c10::cuda::CUDAGuard guard(points.device());
  const int64_t B = scan_ptr ? scan_ptr->size(0) - 1 : 1;
  Tensor scan;
  if (scan_ptr && scan_ptr->is_cuda()) {
    scan = scan_ptr->to(points.device(), at::kInt).contiguous();
  } else {     // a few host integers, by way of pinned memory: a copy from pageable memory would wait for the stream
    Tensor host = at::empty({B + 1}, at::TensorOptions().dtype(at::kInt).pinned_memory(true));
    if (scan_ptr) {
      host.copy_(*scan_ptr);
    } else {
      ints(host)[0] = 0;
      ints(host)[1] = (int32_t)n;
    }
    scan = host.to(points.device(), /*non_blocking=*/true);
  }
  sph_voxel_grid grid;
  grid.B = (int32_t)B;
  for (int i = 0; i < 3; ++i) grid.cells[i] = (int32_t)cells.at(i);
  for (int i = 0; i < 6; ++i) grid.range[i] = (float)range.at(i);
  grid.max_points = (int32_t)max_points;
  grid.max_voxels = (int32_t)max_voxels;
  grid.append_mode = (int32_t)append_mode;
  const int64_t features = check(abi.sph_voxel_feature_count((int32_t)points.size(1), (int)append_mode));
  Tensor scratch = empty({check(abi.sph_voxelize_scratch_bytes(&grid, n))}, at::kByte, points);
  Tensor z_ptr = empty({B, cells[2], cells[1]}, at::kInt, points);
  int32_t nnz = 0;
  const auto* sys_data = static_cast<const float*>(ptr(sys));
  const cudaStream_t st = stream_of(points);
  {
    py::gil_scoped_release release;
    check(abi.sph_voxelize_count(sys_data, ints(scan), n, &grid, ptr(scratch), ints(z_ptr), &nnz, st));
  }
  Tensor feature = empty({nnz, features}, at::kFloat, points), z_idx = empty({nnz}, at::kInt, points);
  Tensor coords, num;
  if (with_coordinates) {
    coords = empty({nnz, 4}, at::kInt, points);
    num = empty({nnz}, at::kInt, points);
  }
  check(abi.sph_voxelize_fill(static_cast<const float*>(ptr(points)), (int32_t)points.size(1), sys_data, ints(scan), n, &grid,
                              ptr(scratch), nnz, static_cast<float*>(ptr(feature)), ints(z_idx),
                              with_coordinates ? ints(coords) : nullptr, with_coordinates ? ints(num) : nullptr, st));
  return py::make_tuple(feature, z_idx, z_ptr, or_none(coords), or_none(num));
}

}  // namespace

PYBIND11_MODULE(sph_host, m) {
  py::class_<ListsReady, std::shared_ptr<ListsReady>>(m, "ListsReady").def("join", &ListsReady::join);
  py::class_<Pending, std::shared_ptr<Pending>>(m, "Pending");
  m.def("load", &load);
  m.def("status_tensor", &status_tensor);
  m.def("side_stream", [](int device) { return (int64_t)side_stream(device).stream(); });
  m.def("rules_subm", &rules_subm);
  m.def("strided_begin", &strided_begin);
  m.def("strided_rules", &strided_rules);
  m.def("lists_of_table", &lists_of_table);
  m.def("exact_lists", &exact_lists);
  m.def("rules_to_nbr", &rules_to_nbr);
  m.def("pack_weight", &pack_weight);
  m.def("conv_gather", &conv_gather);
  m.def("conv_wgrad", &conv_wgrad);
  m.def("epilogue_backward", &epilogue_backward);
  m.def("conv_layer", &conv_layer);
  m.def("init_tensor", &init_tensor);
  m.def("gather_rows", &gather_rows);
  m.def("dense_channels_first", &dense_channels_first);
  m.def("voxel_transform", &voxel_transform);
  m.def("voxelize", &voxelize);
}
