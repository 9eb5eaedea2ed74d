// What the kernels over staged runs of input rows share (conv_strip.cuh, conv_wgrad_strip.cu): fragment loads, products, and
// the runs themselves - which consecutive input rows the entries of a tile lie in, and how they reach shared memory.
#pragma once
#include "common.cuh"
#include "tc_common.cuh"

#include <climits>

namespace sph {
namespace strip {

using tc::cp_async_16;
using tc::cp_async_wait_all;
using tc::smem_u32;

constexpr int kZeroUnits = 8;             // a row of zeros at the start of the buffers, in 16-byte units

template <int DT>
__device__ __forceinline__ void mma_step(uint32_t (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  if constexpr (DT == SPH_I8) {
    asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3},{%4,%5,%6,%7},{%8,%9},{%0,%1,%2,%3};"
                 : "+r"(d[0]), "+r"(d[1]), "+r"(d[2]), "+r"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
  } else if constexpr (DT == SPH_BF16) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3},{%4,%5,%6,%7},{%8,%9},{%0,%1,%2,%3};"
                 : "+r"(d[0]), "+r"(d[1]), "+r"(d[2]), "+r"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
  } else {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3},{%4,%5,%6,%7},{%8,%9},{%0,%1,%2,%3};"
                 : "+r"(d[0]), "+r"(d[1]), "+r"(d[2]), "+r"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
  }
}

// Four 8 x 16-byte matrices: rows 0-7 and 8-15 of a 16-row tile, first and second half of a 32-byte step.
__device__ __forceinline__ void ldmatrix4(uint32_t (&a)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(a[0]), "=r"(a[1]), "=r"(a[2]), "=r"(a[3]) : "r"(addr));
}

// The same with every 8 x 8 matrix of 16-bit values transposed.
__device__ __forceinline__ void ldmatrix4_trans(uint32_t (&a)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(a[0]), "=r"(a[1]), "=r"(a[2]), "=r"(a[3]) : "r"(addr));
}

// Two windows of consecutive input rows, held one behind the other in a buffer.
struct Windows {
  int base1, len1, base2, len2;
  bool fit;
};

// Merges the warps' runs (lo, hi of either part; lo > hi: empty); called by whole warps.
template <int WARPS>
__device__ __forceinline__ Windows merge_runs(const int4* runs, int cap) {
  const int4 mine = runs[threadIdx.x % WARPS];
  const int all_lo = __reduce_min_sync(0xffffffffu, mine.x);
  const int all_hi = __reduce_max_sync(0xffffffffu, max(mine.y, mine.w));
  Windows o;
  o.base1 = all_hi < 0 ? 0 : all_lo;
  o.len1 = all_hi < 0 ? 0 : all_hi - all_lo + 1;
  o.base2 = o.len2 = 0;
  o.fit = true;
  if (o.len1 <= cap) return o;
  // the end of a line of columns lies inside the tile: two windows
  int lo1 = INT_MAX, hi1 = -1, lo2 = INT_MAX, hi2 = -1;
  bool fit = true;
  const int slack = cap / 4;
  auto add = [&](int lo, int hi) {
    if (lo > hi) return;
    if (hi1 < 0 || (lo <= hi1 + slack && hi >= lo1 - slack)) {
      lo1 = min(lo1, lo);
      hi1 = max(hi1, hi);
    } else if (hi2 < 0 || (lo <= hi2 + slack && hi >= lo2 - slack)) {
      lo2 = min(lo2, lo);
      hi2 = max(hi2, hi);
    } else {
      fit = false;
    }
  };
#pragma unroll 1
  for (int w = 0; w < WARPS; ++w) {
    const int4 r = runs[w];
    add(r.x, r.y);
    add(r.z, r.w);
  }
  o.base1 = lo1;
  o.len1 = hi1 - lo1 + 1;
  o.base2 = hi2 < 0 ? 0 : lo2;
  o.len2 = hi2 < 0 ? 0 : hi2 - lo2 + 1;
  o.fit = fit && (int64_t)o.len1 + o.len2 <= cap;
  return o;
}

__device__ __forceinline__ void cp_async_8(uint32_t dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst), "l"(src));
}
__device__ __forceinline__ void cp_async_4(uint32_t dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src));
}

// Channels [c0, c0 + n) of 16-bit rows of an ODD number of channels -> rows `pitch` 16-byte units apart.  A row may start in
// the middle of a word, so nothing wider than an element can be copied as it is: the run is read as the stream of words it
// is, eight in flight per thread, and stored element by element.  `rows` is 4-byte aligned; `total` = elements behind it.
// Not inlined: its loads in flight would cost the kernels registers they need elsewhere.
template <int THREADS>
__device__ __noinline__ void copy_odd_rows(const uint16_t* rows, int64_t total, int base, int len, int channels, int c0, int n,
                                              int pitch, uint32_t to) {
  const int64_t first = (int64_t)base * channels, word0 = first >> 1;
  const int elems = len * channels, words = (int)(((first + elems + 1) >> 1) - word0);
  const int skew = (int)(first & 1);
  const unsigned magic = 0xffffffffu / (unsigned)channels + 1u;        // exact for fewer than 2^26 elements of up to 64 channels
  for (int u0 = threadIdx.x; u0 < words; u0 += THREADS * 8) {
    uint32_t v[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int64_t w = word0 + u0 + i * THREADS;
      if (u0 + i * THREADS < words)
        v[i] = 2 * w + 1 < total ? __ldg((const uint32_t*)rows + w) : (uint32_t)__ldg(rows + 2 * w);
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int e0 = 2 * (u0 + i * THREADS) - skew;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int e = e0 + h;
        if (e < 0 || e >= elems) continue;
        const int r = channels == 1 ? e : (int)__umulhi((unsigned)e, magic), c = e - r * channels - c0;
        if ((unsigned)c < (unsigned)n)
          asm volatile("st.shared.u16 [%0], %1;" ::"r"(to + r * pitch * 16 + c * 2), "h"((uint16_t)(v[i] >> (16 * h))) : "memory");
      }
    }
  }
}

// Rows of a width that is no multiple of 16 bytes -> rows `pitch` units apart, in the widest pieces that keep both sides
// aligned.
template <int THREADS>
__device__ __forceinline__ void copy_ragged_rows(const uint8_t* rows, int64_t n_rows, int base, int len, int row_bytes, int pitch,
                                                 uint32_t to) {
  if ((row_bytes & 3) == 2) {
    copy_odd_rows<THREADS>((const uint16_t*)rows, n_rows * (row_bytes / 2), base, len, row_bytes / 2, 0, row_bytes / 2, pitch, to);
    return;
  }
  const int piece = row_bytes & 1 ? 1 : row_bytes & 4 ? 4 : 8;
  const unsigned per = row_bytes / piece, n = per * len;
  for (unsigned u = threadIdx.x; u < n; u += THREADS) {
    const unsigned r = u / per, b = u % per * piece;
    const uint8_t* src = rows + (int64_t)(base + (int)r) * row_bytes + b;
    const uint32_t dst = to + r * pitch * 16 + b;
    if (piece == 8) cp_async_8(dst, src);
    else if (piece == 4) cp_async_4(dst, src);
    else asm volatile("{.reg .b16 t; cvt.u16.u32 t, %1; st.shared.u8 [%0], t;}" ::"r"(dst), "r"((uint32_t)__ldg(src)) : "memory");
  }
}

// One row of any width, by one thread, in the widest pieces that both sides allow (rows of a multiple of 16 bytes are 16-byte
// aligned, and so on down).
__device__ __forceinline__ void copy_ragged_row(const uint8_t* src, int bytes, uint32_t dst) {
  if ((bytes & 15) == 0) {
    for (int b = 0; b < bytes; b += 16) cp_async_16(dst + b, src + b, 16u);
  } else if ((bytes & 7) == 0) {
    for (int b = 0; b < bytes; b += 8) cp_async_8(dst + b, src + b);
  } else if ((bytes & 3) == 0) {
    for (int b = 0; b < bytes; b += 4) cp_async_4(dst + b, src + b);
  } else if ((bytes & 1) == 0) {
#pragma unroll 4
    for (int b = 0; b < bytes; b += 2)
      asm volatile("st.shared.u16 [%0], %1;" ::"r"(dst + b), "h"(__ldg((const uint16_t*)(src + b))) : "memory");
  } else {
#pragma unroll 4
    for (int b = 0; b < bytes; ++b)
      asm volatile("{.reg .b16 t; cvt.u16.u32 t, %1; st.shared.u8 [%0], t;}" ::"r"(dst + b), "r"((uint32_t)__ldg(src + b)) : "memory");
  }
}

}  // namespace strip
}  // namespace sph
