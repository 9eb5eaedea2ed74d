// extern "C" entry points that are pure dispatch (declared in include/sphconv_b200.h).
#include <stdarg.h>
#include <string.h>

#include <atomic>

#include "common.cuh"

namespace sph {

static thread_local char g_err[512] = "";
static std::atomic<long long> g_launches{0};

void note_launch() { g_launches.fetch_add(1, std::memory_order_relaxed); }

void set_error(const char* fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(g_err, sizeof(g_err), fmt, ap);
  va_end(ap);
}

int current_sm_count() {
  constexpr int kMaxDev = 64;
  static std::atomic<int> s_sms[kMaxDev];     // zero-initialised; a racing first call writes the same value twice
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) {
    set_error("current_sm_count: cudaGetDevice failed");
    return 0;
  }
  int n = (dev >= 0 && dev < kMaxDev) ? s_sms[dev].load(std::memory_order_relaxed) : 0;
  if (n == 0) {
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) {
      set_error("current_sm_count: cudaDeviceGetAttribute failed");
      return 0;
    }
    if (dev >= 0 && dev < kMaxDev) s_sms[dev].store(n, std::memory_order_relaxed);
  }
  return n;
}

// conv_generic.cu
int conv_gather_generic(const void* rows, int64_t n_rows, const void* weight, const int* nbr, int64_t n_out, int kv,
                        int K, int N, int flip_k, const float* scale, const float* bias, int relu, void* out,
                        int out_dtype, int* status, cudaStream_t st);
// conv_ffma.cu
int conv_gather_ffma(const void* rows, int dtype, int64_t n_rows, const void* weight, const int* nbr, int64_t n_out,
                     int kv, int K, int N, int flip_k, const float* scale, Bias bias, int relu, void* out,
                     int out_dtype, int* status, cudaStream_t st);
int conv_wgrad_ffma(const void* rows, const void* dout, int dtype, int64_t n_rows, const int* nbr, int64_t n_out, int kv,
                    int K, int N, float* dw, int* status, cudaStream_t st);
// conv_tc.cu
int conv_gather_tc(const void* rows, int dtype, int64_t n_rows, const void* packed, const int* nbr, int64_t n_out,
                   int kv, int K, int N, int flip_k, const float* scale, Bias bias, int relu, void* out,
                   int out_dtype, int* status, cudaStream_t st);
bool conv_tc_supported(int dtype, int kv, int K, int N);
int64_t packed_weight_bytes(int dtype, int kv, int K, int N);
int pack_weight(const void* w, int dtype, int kv, int K, int N, void* packed, cudaStream_t st);
// conv_tc_rows.cu
bool conv_tc_rows_supported(int dtype, int kv, int K, int N);
int conv_gather_tc_rows(const void* rows, int dtype, int64_t n_rows, const void* packed, const int* nbr, int64_t n_out,
                        int kv, int K, int N, int flip_k, const float* scale, Bias bias, int relu, void* out,
                        int out_dtype, int* status, cudaStream_t st);
// conv_tmem.cu
bool conv_tmem_supported(int dtype, int kv, int K, int N);
int conv_gather_tmem(const void* rows, int dtype, int64_t n_rows, const void* packed, const int* nbr, int64_t n_out, int kv,
                     int K, int N, int flip_k, const float* scale, Bias bias, int relu, void* out, int out_dtype, int* status,
                     cudaStream_t st);
// conv_strip.cu
bool conv_strip_supported(int dtype, int kv, int K, int N);
int64_t strip_filter_bytes(int dtype, int kv, int K, int N);
int pack_strip_filter(const void* w, int dtype, int kv, int K, int N, void* packed, cudaStream_t st);
int conv_gather_strip(const void* rows, int dtype, int64_t n_rows, const void* packed, const int* nbr, int64_t n_out, int kv,
                    int K, int N, int flip_k, const float* scale, Bias bias, int relu, void* out, int out_dtype,
                    int* status, cudaStream_t st);
// conv_sparse.cu
bool conv_sparse_supported(int dtype, int kv, int K, int N);
int conv_gather_sparse(const void* rows, int dtype, int64_t n_rows, const void* weight, const int* nbr, int64_t n_out,
                       int kv, int K, int N, int flip_k, const float* scale, Bias bias, int relu, void* out,
                       int out_dtype, int* status, cudaStream_t st);

bool conv_wgrad_pairs_supported(int dtype, int kv, int K, int N);
int conv_wgrad_pairs(const void* rows, const void* dout, int dtype, int64_t n_rows, const int* nbr, int64_t n_out,
                     int kv, int K, int N, float* dw, int* status, cudaStream_t st);

// conv_wgrad_strip.cu
bool conv_wgrad_strip_supported(int dtype, int K, int N);
int conv_wgrad_strip(const void* rows, const void* dout, int dtype, int64_t n_rows, const int* nbr, int64_t n_out, int kv,
                     int K, int N, float* dw, int* status, cudaStream_t st);
// conv_wgrad_tc.cu
bool conv_wgrad_tc_supported(int dtype, int kv, int K, int N);
int conv_wgrad_tc(const void* rows, const void* dout, int dtype, int64_t n_rows, const int* nbr, int64_t n_out, int kv,
                  int K, int N, float* dw, int* status, cudaStream_t st);

}  // namespace sph

using namespace sph;

extern "C" const char* sph_last_error(void) { return g_err; }
extern "C" int sph_version(void) { return 100; }
extern "C" int64_t sph_kernel_launches(void) { return (int64_t)g_launches.load(std::memory_order_relaxed); }

// Whether a shape runs the strip kernel (conv_strip.cuh) when the caller passes a packed filter: everything the tcgen05
// kernels do not take, but for rows of 4 or 8 channels (sparse first layers: the pair kernel); of what they do take, 16
// channels to at most 16 (1.1 to 1.4 times faster at 1.5 to 12 neighbours per row; from 32 output channels on it loses).
static bool runs_strip(int dtype, int kv, int K, int N) {
  if (!conv_strip_supported(dtype, kv, K, N)) return false;
  if (conv_tc_supported(dtype, kv, K, N)) return dtype != SPH_I8 && K == 16 && N <= 16;
  return !((K == 4 || K == 8) && conv_sparse_supported(dtype, kv, K, N));
}

extern "C" int64_t sph_packed_weight_bytes(int dtype, int32_t kv, int32_t k_ch, int32_t n_ch) {
  if (runs_strip(dtype, kv, k_ch, n_ch)) return strip_filter_bytes(dtype, kv, k_ch, n_ch);
  if (!conv_tc_supported(dtype, kv, k_ch, n_ch)) return 0;
  return packed_weight_bytes(dtype, kv, k_ch, n_ch);
}

extern "C" int sph_pack_weight(const void* d_weight, int dtype, int32_t kv, int32_t k_ch, int32_t n_ch,
                               void* d_packed, void* stream) {
  SPH_CHECK_ARG(d_weight && d_packed, "null pointer");
  if (runs_strip(dtype, kv, k_ch, n_ch)) return pack_strip_filter(d_weight, dtype, kv, k_ch, n_ch, d_packed, (cudaStream_t)stream);
  return pack_weight(d_weight, dtype, kv, k_ch, n_ch, d_packed, (cudaStream_t)stream);
}

extern "C" int sph_conv_uses_tensor_cores(int dtype, int32_t k_ch, int32_t n_ch) {
  return conv_tc_supported(dtype, 27, k_ch, n_ch) ? 1 : 0;
}

extern "C" int sph_conv_uses_pair_kernel(int dtype, int32_t k_ch, int32_t n_ch) {
  return (!conv_tc_supported(dtype, 27, k_ch, n_ch) && conv_sparse_supported(dtype, 27, k_ch, n_ch)) ? 1 : 0;
}

extern "C" int sph_conv_wgrad_kernel(int dtype, int32_t k_ch, int32_t n_ch) {
  if (conv_wgrad_tc_supported(dtype, 27, k_ch, n_ch)) return 1;
  return conv_wgrad_pairs_supported(dtype, 27, k_ch, n_ch) ? 2 : 0;
}

// The kernels that run; sph_conv_gather and sph_conv_wgrad switch on these.  packed: the caller passes the filter's image and all
// operands are 16-byte aligned; aligned: the operands the kernel reads are (words: 4-byte aligned).
static int gather_kernel(int dtype, int kv, int K, int N, bool packed, bool aligned) {
  if (packed && runs_strip(dtype, kv, K, N)) return SPH_KERNEL_STRIP;
  // 64-byte rows: the form with the output row on the TMEM lane (absent neighbours masked, not copied) is the faster
  // of the two; wider rows are dense deep layers, where the transposed form issues half as many instructions
  if (packed && K * dtype_bytes(dtype) == 64 && conv_tc_rows_supported(dtype, kv, K, N)) return SPH_KERNEL_TC_ROWS;
  if (packed && conv_tc_supported(dtype, kv, K, N)) return SPH_KERNEL_TC;
  // narrow rows the tensor-core kernels do not take (the first layer of an encoder: 4 or 8 channels in, a sparse level;
  // int8 rows of up to 16 channels) and small fp32 layers: the pair-compacting kernel (faster than the row-walking one from 1 to
  // 22 neighbours per row)
  if (aligned && conv_sparse_supported(dtype, kv, K, N)) return SPH_KERNEL_PAIRS;
  return SPH_KERNEL_GENERAL;
}

static int wgrad_kernel(int dtype, int kv, int K, int N, bool aligned, bool words) {
  // the pairs' kernel up to 2048 gradients an offset (1.1 to 3 times faster than the tcgen05 kernel from 1.5 to 12 pairs a row);
  // at 64 x 64, the deep and dense levels, the tcgen05 kernel (22 pairs of 27: 0.70 against 1.19 ms on 1.4 M rows), and where fewer
  // than nine offsets leave the former's warps idle (3 x 1 x 1: 32 -> 32 on 525 k rows 46 against 107 us)
  const bool tc = aligned && conv_wgrad_tc_supported(dtype, kv, K, N);
  if (words && conv_wgrad_strip_supported(dtype, K, N) && ((K * N <= 2048 && kv >= 9) || !tc)) return SPH_KERNEL_STRIP;
  if (tc) return SPH_KERNEL_TC;
  // small fp32 layers: the pair-compacting walk
  if (dtype == SPH_F32 && aligned && conv_wgrad_pairs_supported(dtype, kv, K, N)) return SPH_KERNEL_PAIRS;
  return SPH_KERNEL_GENERAL;
}

extern "C" int sph_conv_kernel(int dtype, int32_t kv, int32_t k_ch, int32_t n_ch, int wgrad) {
  SPH_CHECK_ARG(dtype >= SPH_F32 && dtype <= SPH_I8 && kv > 0 && k_ch > 0 && n_ch > 0, "bad sizes");
  return wgrad ? wgrad_kernel(dtype, kv, k_ch, n_ch, true, true) : gather_kernel(dtype, kv, k_ch, n_ch, true, true);
}

extern "C" int sph_conv_uses_tmem(int dtype, int32_t kv, int32_t k_ch, int32_t n_ch) {
  const int kernel = sph_conv_kernel(dtype, kv, k_ch, n_ch, 0);
  return (kernel == SPH_KERNEL_TC || kernel == SPH_KERNEL_TC_ROWS) && conv_tmem_supported(dtype, kv, k_ch, n_ch) ? 1 : 0;
}

static bool out_dtype_ok(int dtype, int out_dtype) {
  if (out_dtype < SPH_F32 || out_dtype > SPH_I8) return false;
  if (out_dtype == SPH_I8 && dtype != SPH_I8) return false;
  return true;
}

extern "C" int sph_conv_gather(const void* d_rows, int dtype, int64_t n_rows, const void* d_weight,
                               const void* d_packed, const int32_t* d_nbr, int64_t n_out, int32_t kv, int32_t k_ch,
                               int32_t n_ch, int flip_k, const float* d_scale, const void* d_bias, int relu,
                               void* d_out, int out_dtype, int32_t* d_status, void* stream) {
  SPH_CHECK_ARG(n_rows >= 0 && n_out >= 0 && kv > 0 && k_ch > 0 && n_ch > 0, "bad sizes");
  SPH_CHECK_ARG(dtype >= SPH_F32 && dtype <= SPH_I8, "unknown dtype");
  SPH_CHECK_ARG(out_dtype_ok(dtype, out_dtype), "unsupported output dtype for this input dtype");
  if (n_out == 0) return SPH_OK;
  SPH_CHECK_ARG(d_nbr && d_out && (d_weight || d_packed), "null pointer");
  SPH_CHECK_ARG(n_rows == 0 || d_rows, "null rows");
  SPH_CHECK_ARG(n_rows < 0x7fffffffLL && n_out < 0x7fffffffLL, "row ids are 32-bit");
  const bool bias_16 = relu & SPH_BIAS_IN_ROW_TYPE;
  relu = (relu & ~SPH_BIAS_IN_ROW_TYPE) != 0;
  SPH_CHECK_ARG(!bias_16 || dtype == SPH_F16 || dtype == SPH_BF16, "a bias in the rows' type needs 16-bit rows");
  const Bias bias = {d_bias, bias_16 ? dtype : SPH_F32};
  cudaStream_t st = (cudaStream_t)stream;
  // the tensor-core kernels copy 16 bytes at a time
  const bool packed = d_packed && (((uintptr_t)d_rows | (uintptr_t)d_packed | (uintptr_t)d_out) & 15u) == 0;
  const bool aligned = (((uintptr_t)d_rows | (uintptr_t)d_weight | (uintptr_t)d_out) & 15u) == 0;
  const int kernel = gather_kernel(dtype, kv, k_ch, n_ch, packed, aligned);
  SPH_CHECK_ARG(d_weight || (kernel != SPH_KERNEL_PAIRS && kernel != SPH_KERNEL_GENERAL),
                "the CUDA-core kernels need the unpacked weight");
  // 9 or 27 offsets and up to 64 channels out: the rows by way of tensor memory (conv_tmem.cu), against the two forms that gather into
  // shared memory (us, launches one behind the other, 16-bit rows):
  //   submanifold 32 -> 32, 61 k / 1.5 M rows 23 -> 16 / 324 -> 194, 64 -> 64, 22 k / 683 k rows 21 -> 17 / 248 -> 165;
  //   input gradients of strided layers 64 -> 32, 1.5 M rows 510 -> 185, 32 -> 16, 567 k rows 113 -> 83;
  //   strided 16 -> 32, 61 k / 1.5 M rows 19 -> 16 / 197 -> 164, 32 -> 64, 22 k / 683 k rows 17.0 -> 16.6 / 179 -> 118;
  //   9 x 3 x 1 filters, whose lines span three heights, 32 -> 32, 228 k rows 57 -> 51.
  // It does not win where most rows lie beyond the runs' buffers: 64 -> 64 on volumes 95 % full at 256 depths, submanifold 190 -> 202,
  // strided 36 -> 44; tables without locality, 300 k rows, 16 -> 32 56 -> 58, 32 -> 32 71 -> 78, 64 -> 64 112 -> 132, 1.5 M rows 575 -> 763.
  // The sizes that the call knows do not tell these from the others, and the rows of this library's own tables are numbered along the
  // grid.  Without rows there is nothing to describe to TMA.
  if ((kernel == SPH_KERNEL_TC || kernel == SPH_KERNEL_TC_ROWS) && n_rows > 0 && conv_tmem_supported(dtype, kv, k_ch, n_ch))
    return conv_gather_tmem(d_rows, dtype, n_rows, d_packed, d_nbr, n_out, kv, k_ch, n_ch, flip_k, d_scale, bias, relu, d_out,
                            out_dtype, d_status, st);
  switch (kernel) {
    case SPH_KERNEL_STRIP:
      return conv_gather_strip(d_rows, dtype, n_rows, d_packed, d_nbr, n_out, kv, k_ch, n_ch, flip_k, d_scale, bias, relu,
                               d_out, out_dtype, d_status, st);
    case SPH_KERNEL_TC_ROWS:
      return conv_gather_tc_rows(d_rows, dtype, n_rows, d_packed, d_nbr, n_out, kv, k_ch, n_ch, flip_k, d_scale, bias, relu,
                                 d_out, out_dtype, d_status, st);
    case SPH_KERNEL_TC:
      return conv_gather_tc(d_rows, dtype, n_rows, d_packed, d_nbr, n_out, kv, k_ch, n_ch, flip_k, d_scale, bias, relu, d_out,
                            out_dtype, d_status, st);
    case SPH_KERNEL_PAIRS:
      return conv_gather_sparse(d_rows, dtype, n_rows, d_weight, d_nbr, n_out, kv, k_ch, n_ch, flip_k, d_scale, bias, relu,
                                d_out, out_dtype, d_status, st);
  }
  if (dtype == SPH_I8)
    return conv_gather_generic(d_rows, n_rows, d_weight, d_nbr, n_out, kv, k_ch, n_ch, flip_k, d_scale, (const float*)d_bias, relu,
                               d_out, out_dtype, d_status, st);
  return conv_gather_ffma(d_rows, dtype, n_rows, d_weight, d_nbr, n_out, kv, k_ch, n_ch, flip_k, d_scale, bias, relu,
                          d_out, out_dtype, d_status, st);
}

extern "C" int sph_conv_wgrad(const void* d_rows, const void* d_dout, int dtype, int64_t n_rows,
                              const int32_t* d_nbr, int64_t n_out, int32_t kv, int32_t k_ch, int32_t n_ch,
                              float* d_dweight, int zero_init, int32_t* d_status, void* stream) {
  SPH_CHECK_ARG(n_rows >= 0 && n_out >= 0 && kv > 0 && k_ch > 0 && n_ch > 0, "bad sizes");
  SPH_CHECK_ARG(d_dweight, "null gradient buffer");
  cudaStream_t st = (cudaStream_t)stream;
  if (zero_init) SPH_CUDA(cudaMemsetAsync(d_dweight, 0, (size_t)kv * k_ch * n_ch * sizeof(float), st));
  if (n_out == 0 || n_rows == 0) return SPH_OK;
  SPH_CHECK_ARG(d_rows && d_dout && d_nbr, "null pointer");
  const uintptr_t at = (uintptr_t)d_rows | (uintptr_t)d_dout;
  switch (wgrad_kernel(dtype, kv, k_ch, n_ch, (at & 15u) == 0, (at & 3u) == 0)) {
    case SPH_KERNEL_STRIP:
      return conv_wgrad_strip(d_rows, d_dout, dtype, n_rows, d_nbr, n_out, kv, k_ch, n_ch, d_dweight, d_status, st);
    case SPH_KERNEL_TC:
      return conv_wgrad_tc(d_rows, d_dout, dtype, n_rows, d_nbr, n_out, kv, k_ch, n_ch, d_dweight, d_status, st);
    case SPH_KERNEL_PAIRS:
      return conv_wgrad_pairs(d_rows, d_dout, dtype, n_rows, d_nbr, n_out, kv, k_ch, n_ch, d_dweight, d_status, st);
  }
  return conv_wgrad_ffma(d_rows, d_dout, dtype, n_rows, d_nbr, n_out, kv, k_ch, n_ch, d_dweight, d_status, st);
}
