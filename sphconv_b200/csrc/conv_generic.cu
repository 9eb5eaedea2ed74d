// int8 rows of the channel counts that neither the tensor-core kernels nor the pair-compacting kernel take: a thread
// group owns one output row, walks its KV neighbour-table entries and accumulates in 32-bit integers, so there is no
// scatter and no atomic (the reference scatters with read-modify-write per 8 pairs, include/sphconv/iterator.cu.h:1467-1625).
#include "common.cuh"

namespace sph {

namespace {

__device__ __forceinline__ void store_out(void* out, int out_dtype, int64_t idx, float v) {
  switch (out_dtype) {
    case SPH_F32: ((float*)out)[idx] = v; break;
    case SPH_F16: ((__half*)out)[idx] = __float2half_rn(v); break;
    case SPH_BF16: ((__nv_bfloat16*)out)[idx] = __float2bfloat16_rn(v); break;
    default: {
      float r = rintf(v);
      r = fminf(fmaxf(r, -127.f), 127.f);
      ((int8_t*)out)[idx] = (int8_t)(int)r;
    }
  }
}

constexpr int kGenThreads = 128;

// TPR threads per output row, each owning 4 consecutive output channels.
__global__ void __launch_bounds__(kGenThreads)
conv_gather_generic_kernel(const int8_t* __restrict__ rows, int64_t n_rows, const int8_t* __restrict__ weight,
                           const int* __restrict__ nbr, int64_t n_out, int kv, int K, int N, int tpr, int flip_k,
                           const float* __restrict__ scale, const float* __restrict__ bias, int relu,
                           void* __restrict__ out, int out_dtype, int* __restrict__ status) {
  after_previous();
  const int rows_per_block = kGenThreads / tpr;
  const int sub = threadIdx.x % tpr;
  const int64_t r = (int64_t)blockIdx.x * rows_per_block + threadIdx.x / tpr;
  if (r >= n_out) return;
  const int oc0 = sub * 4;
  if (oc0 >= N) return;
  const int noc = min(4, N - oc0);
  int acc[4] = {0, 0, 0, 0};
  for (int k = 0; k < kv; ++k) {
    const int tk = flip_k ? kv - 1 - k : k;
    const int i = __ldg(nbr + (int64_t)tk * n_out + r);
    if (i < 0) continue;
    if (i >= n_rows) {
      if (status) atomicOr(status, SPH_STATUS_BAD_INDEX);
      continue;
    }
    const int8_t* x = rows + (int64_t)i * K;
    const int8_t* w = weight + (int64_t)k * K * N + oc0;
    for (int ic = 0; ic < K; ++ic) {
      const int xv = (int)x[ic];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if (j < noc) acc[j] += xv * (int)w[(int64_t)ic * N + j];
      }
    }
  }
  for (int j = 0; j < noc; ++j) {
    float v = (float)acc[j];
    if (scale) v *= scale[oc0 + j];
    if (bias) v += bias[oc0 + j];
    if (relu) v = fmaxf(v, 0.f);
    store_out(out, out_dtype, r * N + oc0 + j, v);
  }
}

}  // namespace

int conv_gather_generic(const void* rows, int64_t n_rows, const void* weight, const int* nbr, int64_t n_out, int kv,
                        int K, int N, int flip_k, const float* scale, const float* bias, int relu, void* out,
                        int out_dtype, int* status, cudaStream_t st) {
  int tpr = 1;
  while (tpr * 4 < N) tpr <<= 1;
  if (tpr > kGenThreads) {
    set_error("n_ch %d too large for the CUDA-core kernel", N);
    return SPH_ERR_LIMIT;
  }
  const int rows_per_block = kGenThreads / tpr;
  const int64_t blocks = div_up64(n_out, rows_per_block);
  launch(conv_gather_generic_kernel, (unsigned)blocks, kGenThreads, 0, st, (const int8_t*)rows, n_rows, (const int8_t*)weight, nbr, n_out, kv, K, N, tpr, flip_k, scale, bias, relu, out,
      out_dtype, status);
  SPH_LAUNCH_CHECK();
  return SPH_OK;
}

}  // namespace sph
