// Shared helpers of the sphconv_b200 CUDA library (sm_100a only).
#pragma once

#include <cuda_runtime.h>
#include <cuda_fp16.h>
#include <cuda_bf16.h>
#include <stdint.h>
#include <stdio.h>

#include "sphconv_b200.h"

namespace sph {

void set_error(const char* fmt, ...);
void note_launch();  // counts kernels launched by this library (sph_kernel_launches)

#define SPH_CHECK_ARG(cond, msg)                         \
  do {                                                   \
    if (!(cond)) {                                       \
      ::sph::set_error("%s: %s", __func__, msg);         \
      return SPH_ERR_INVALID;                            \
    }                                                    \
  } while (0)

#define SPH_CUDA(call)                                                                   \
  do {                                                                                   \
    cudaError_t e__ = (call);                                                            \
    if (e__ != cudaSuccess) {                                                            \
      ::sph::set_error("%s: %s failed: %s", __func__, #call, cudaGetErrorString(e__));   \
      return SPH_ERR_CUDA;                                                               \
    }                                                                                    \
  } while (0)

#define SPH_LAUNCH_CHECK()                                                               \
  do {                                                                                   \
    cudaError_t e__ = cudaGetLastError();                                                \
    if (e__ != cudaSuccess) {                                                            \
      ::sph::set_error("%s: kernel launch failed: %s", __func__, cudaGetErrorString(e__)); \
      return SPH_ERR_CUDA;                                                               \
    }                                                                                    \
    ::sph::note_launch();                                                                \
  } while (0)

// A kernel of this library may be launched before the one in front of it in the stream has ended (programmatic dependent launch):
// its blocks take their places when the last ones of that kernel have ended, or earlier where that kernel allows it, and
// after_previous(), in front of every access to global memory, holds them until all of it is complete and its writes are visible.
// A chain of small kernels then costs about a microsecond a kernel less (both rule sets of a batch of 3 small scans 117 -> 100 us).
// The wait is in every kernel, also in those that nothing of the library precedes: a kernel that skipped it could complete before
// its predecessor, and its successor would run too early.
// What the kernel in front writes is read behind the wait by __ldg and through const __restrict__ pointers as well: the data does not
// change from there on, but it may have since the block began, so this relies on the compiler leaving read-only loads behind the
// wait, a volatile statement that clobbers memory.  tests/test_gpu_overlap.py has the chains that would show it doing otherwise.
template <typename... Params, typename... Args>
inline void launch(void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, Args&&... args) {
  cudaLaunchAttribute early;
  early.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  early.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t c = {};
  c.gridDim = grid;
  c.blockDim = block;
  c.dynamicSmemBytes = smem;
  c.stream = st;
  c.attrs = &early;
  c.numAttrs = 1;
  (void)cudaLaunchKernelEx(&c, kernel, static_cast<Params>(args)...);      // SPH_LAUNCH_CHECK() reads the error
}
// EARLY: a grid of at most one block per SM lets its successor in at once, which finds room beside it on every SM.  Blocks let in
// beside a larger grid, or at the end of a persistent one, all go to the SMs that are free first: 16 blocks behind a convolution
// took 57 us instead of 9, and behind grids of up to four blocks per SM tables and lists took (us, such grids too / only these) 43 / 27 on 93 k
// rows of 70 scans, 121 / 75 for their strided set, 199 / 132 on 128 k rows 2000 deep.
constexpr unsigned kEarlyBlocks = 148;
template <bool EARLY = true>
__device__ __forceinline__ void after_previous(unsigned most = kEarlyBlocks) {
  if (EARLY && gridDim.x * gridDim.y <= most) asm volatile("griddepcontrol.launch_dependents;");
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

__host__ __device__ inline int div_up(int a, int b) { return (a + b - 1) / b; }
__host__ __device__ inline int64_t div_up64(int64_t a, int64_t b) { return (a + b - 1) / b; }

inline int dtype_bytes(int dtype) {
  switch (dtype) {
    case SPH_F32: return 4;
    case SPH_F16: return 2;
    case SPH_BF16: return 2;
    case SPH_I8: return 1;
    default: return 0;
  }
}

// Multiprocessor count of the CURRENT device (cached per device ordinal, thread-safe); 0 with the error set on failure.
int current_sm_count();

// Geometry in the form the kernels take by value.
struct Geom {
  int B, H, W, D, oH, oW, oD;
  int KH, KW, KD, KV;
  int sH, sW, sD, pH, pW, pD;
  int dH, dW, dD;   // dilation: kernel offset k reads input o*s - p + k*d
  int tH, tW, tgH, tgW, nTile;
};

// Per-channel bias of a convolution's epilogue: float32, or 16-bit values as the parameter holds them (a float32 copy would have
// to be made in every call, or would not see every write to the parameter).
struct Bias {
  const void* data;                 // or null: no bias
  int dtype;                        // SPH_F32, SPH_F16 or SPH_BF16
  // A kernel without 16-bit rows has no 16-bit bias.  The 16-bit load is the builtin one of an integer: that of a __half is
  // an asm statement, which the compiler may move in front of the check for null.
  template <bool MAY_BE_16_BIT>
  __device__ __forceinline__ float at(int c) const {
    if (data == nullptr) return 0.f;
    if (MAY_BE_16_BIT && dtype != SPH_F32) {
      const unsigned short bits = __ldg((const unsigned short*)data + c);
      return dtype == SPH_F16 ? __half2float(__ushort_as_half(bits)) : __uint_as_float((unsigned)bits << 16);
    }
    return __ldg((const float*)data + c);
  }
};

// Allows a kernel `limit` bytes of dynamic shared memory: what all its launches stay within, not what the launch at hand takes.
// Threads launch one kernel with different sizes, and a bound lowered between another thread's call and its launch would
// fail that launch.
template <typename F>
inline cudaError_t allow_smem(F* kernel, int limit) {
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, limit);
}

// Validates and converts; returns SPH_OK or an error code (message set).
int make_geom(const sph_geom* g, Geom* out);

// rules.cu: inclusive prefix over columns of the popcounts of per-column bit masks; the total also goes to a word of mapped
// host memory when total_host is not null.
int column_prefix_from_masks(const uint32_t* mask, int words, int64_t ncols, int* prefix, int* blocksum, int* total_dev,
                             int* total_host, cudaStream_t st);

// rules.cu: a word of mapped pinned host memory of the current device, for a call that waits for what its kernels write there
// (see there), which then gives it back.
struct HostWord {
  int32_t *host, *dev;
};
int take_host_word(HostWord* w);
void give_host_word(const HostWord& w);

}  // namespace sph
