#include "conv_strip.cuh"

namespace sph {
int launch_strip_f16(StripParams& p, const StripShape& s, cudaStream_t st) { return launch_strip<SPH_F16>(p, s, st); }
}  // namespace sph
