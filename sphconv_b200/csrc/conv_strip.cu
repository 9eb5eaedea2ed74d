// Dispatch of the strip kernel (conv_strip.cuh) and its filter image.
#include "common.cuh"
#include "conv_strip.h"

namespace sph {

namespace {

// [KV][K][N] filter -> the image the kernel reads: unit ((k * KS + s) * NT/2 + n/2) * 32 + lane holds, for the lane's output
// channel 8n + lane/4 (and 8(n+1) + lane/4), the 4 bytes of input channels at byte 32s + 4t of a row and the 4 at 32s + 16 + 4t
// (t = lane % 4): the B fragments of two instructions.  Zeros beyond K and N.
template <typename T>
__global__ void pack_strip_kernel(const T* __restrict__ w, int kv, int K, int N, int ks, int nt, uint4* __restrict__ image) {
  after_previous();
  const int64_t u = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int per_k = ks * (nt / 2) * 32;
  if (u >= (int64_t)kv * per_k) return;
  const int k = (int)(u / per_k), rest = (int)(u % per_k);
  const int lane = rest % 32, pair = rest / 32 % (nt / 2), s = rest / 32 / (nt / 2);
  constexpr int PER = 4 / (int)sizeof(T);
  union { T v[4 * PER]; uint4 q; } o;
#pragma unroll
  for (int h = 0; h < 4; ++h)
#pragma unroll
    for (int j = 0; j < PER; ++j) {
      const int c = (s * 32 + (h & 1) * 16 + (lane & 3) * 4) / (int)sizeof(T) + j, n = (pair * 2 + (h >> 1)) * 8 + (lane >> 2);
      o.v[h * PER + j] = (c < K && n < N) ? w[((int64_t)k * K + c) * N + n] : T(0);
    }
  image[u] = o.q;
}

struct Plan {
  int ks, nt, units;
  bool whole;
};

bool plan(int dtype, int kv, int K, int N, Plan* o) {
  if (dtype != SPH_F16 && dtype != SPH_BF16 && dtype != SPH_I8) return false;
  const int row_bytes = K * dtype_bytes(dtype);
  if (row_bytes > 128 || N > 64 || N < 1 || kv < 1) return false;
  o->whole = row_bytes == 32 || row_bytes == 64 || row_bytes == 128;
  o->ks = row_bytes <= 32 ? 1 : row_bytes <= 64 ? 2 : 4;
  o->nt = N <= 16 ? 2 : N <= 32 ? 4 : 8;
  const int64_t units = (int64_t)kv * o->ks * (o->nt / 2) * 32;
  // the filter and two buffers of 320 input rows (a tile of 256 output rows and the columns at its edges)
  if (units * 16 + 1024 + 2 * 320 * ((row_bytes + 15) / 16 | 1) * 16 > kStripSmem) return false;
  o->units = (int)units;
  return true;
}

}  // namespace

bool conv_strip_supported(int dtype, int kv, int K, int N) {
  Plan s;
  return plan(dtype, kv, K, N, &s);
}

int64_t strip_filter_bytes(int dtype, int kv, int K, int N) {
  Plan s;
  return plan(dtype, kv, K, N, &s) ? (int64_t)s.units * 16 : 0;
}

int pack_strip_filter(const void* w, int dtype, int kv, int K, int N, void* packed, cudaStream_t st) {
  Plan s;
  if (!plan(dtype, kv, K, N, &s)) {
    set_error("pack_strip_filter: unsupported dtype/shape");
    return SPH_ERR_UNSUPPORTED;
  }
  const unsigned blocks = (unsigned)div_up(s.units, 256);
  if (dtype == SPH_I8) launch(pack_strip_kernel<int8_t>, blocks, 256, 0, st, (const int8_t*)w, kv, K, N, s.ks, s.nt, (uint4*)packed);
  else launch(pack_strip_kernel<uint16_t>, blocks, 256, 0, st, (const uint16_t*)w, kv, K, N, s.ks, s.nt, (uint4*)packed);
  SPH_LAUNCH_CHECK();
  return SPH_OK;
}

int conv_gather_strip(const void* rows, int dtype, int64_t n_rows, const void* packed, const int* nbr, int64_t n_out, int kv,
                      int K, int N, int flip_k, const float* scale, Bias bias, int relu, void* out, int out_dtype,
                      int* status, cudaStream_t st) {
  Plan s;
  if (!plan(dtype, kv, K, N, &s)) {
    set_error("conv_gather_strip: unsupported dtype/shape");
    return SPH_ERR_UNSUPPORTED;
  }
  if (((uintptr_t)rows | (uintptr_t)packed | (uintptr_t)out) & 15u) {
    set_error("conv_gather_strip: rows, filter image and output must be 16-byte aligned");
    return SPH_ERR_INVALID;
  }
  StripParams p;
  p.rows = (const uint8_t*)rows; p.filter = (const uint4*)packed; p.nbr = nbr;
  p.n_rows = n_rows; p.n_out = n_out;
  p.kv = kv; p.N = N; p.row_bytes = K * dtype_bytes(dtype); p.flip_k = flip_k; p.relu = relu; p.out_dtype = out_dtype;
  p.scale = scale; p.bias = bias; p.out = out; p.status = status;
  p.filter_units = s.units;
  StripShape shape;
  shape.ks = s.ks; shape.nt = s.nt; shape.whole = s.whole;
  switch (dtype) {
    case SPH_F16: return launch_strip_f16(p, shape, st);
    case SPH_BF16: return launch_strip_bf16(p, shape, st);
    default: return launch_strip_i8(p, shape, st);
  }
}

}  // namespace sph
