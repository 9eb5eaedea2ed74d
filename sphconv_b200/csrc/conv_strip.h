// Launch parameters of the strip kernel (conv_strip.cuh), shared by its per-type files and the dispatch (conv_strip.cu).
#pragma once
#include <stdint.h>

#include "common.cuh"

namespace sph {

constexpr int kStripThreads = 256;

struct StripParams {
  const uint8_t* rows;
  const uint4* filter;                    // packed image
  const int* nbr;                         // [KV, n_out]
  int64_t n_rows, n_out;
  int kv, N, row_bytes, flip_k, relu, out_dtype;
  const float* scale;
  Bias bias;
  void* out;
  int* status;
  int filter_units;                       // 16-byte units of the image
  int tiles;                              // tiles of the launch
  int cap;                                // input rows a buffer holds
};

// Steps of 32 bytes, 8-channel tiles of the output; whole: rows are exactly 32 * ks bytes.
struct StripShape {
  int ks, nt;
  bool whole;
};

constexpr int kStripSmem = 222 * 1024;    // dynamic shared memory of a CTA at most
inline int strip_fixed_bytes(int filter_units) { return filter_units * 16 + 128 + 2 * 8 * 16 + 128; }

int launch_strip_f16(StripParams& p, const StripShape& s, cudaStream_t st);
int launch_strip_bf16(StripParams& p, const StripShape& s, cudaStream_t st);
int launch_strip_i8(StripParams& p, const StripShape& s, cudaStream_t st);

}  // namespace sph
