#include "conv_strip.cuh"

namespace sph {
int launch_strip_i8(StripParams& p, const StripShape& s, cudaStream_t st) { return launch_strip<SPH_I8>(p, s, st); }
}  // namespace sph
