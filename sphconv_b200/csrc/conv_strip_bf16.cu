#include "conv_strip.cuh"

namespace sph {
int launch_strip_bf16(StripParams& p, const StripShape& s, cudaStream_t st) { return launch_strip<SPH_BF16>(p, s, st); }
}  // namespace sph
