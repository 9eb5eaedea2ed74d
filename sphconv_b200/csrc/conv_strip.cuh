// Gather-GEMM over strips of input rows (mma.sync + ldmatrix): 16-bit and int8 rows of up to 128 bytes, up to 64 output
// channels, filters that stay in shared memory.  Included once per element type (conv_strip_*.cu).
//
//   out[r,:] = epilogue( sum_k rows[nbr[k][r], :] @ W[k] )          r in [0, n_out)
//
// Rows are numbered along the columns of the grid, so the neighbours that consecutive output rows have in one line of
// columns - the 9 offsets of one kernel height - lie in ONE short run of consecutive input rows (two at the end of a line).
// A tcgen05 kernel has to bring every pair's row to shared memory once per offset in the order of the output rows: 12 to
// 22 row copies per output row that the shared-memory pipe is busy with, handed over through barriers.  Here the run is
// copied once and ldmatrix picks the rows out of it: its 16-byte pieces are addressed lane by lane, so the gather IS the
// operand load.  At these widths nothing is lost on the tensor side: a tcgen05.mma of N <= 64 takes ~60 cycles whatever it
// multiplies, which is the rate of mma.sync (1024 multiply-adds a cycle and SM).  Rows of any width go through it.
//
//  * a CTA (8 warps) owns 256 consecutive output rows x all output channels, accumulators in registers, and walks
//    the offsets in groups of 9: table entries of the group after next in flight, the next group's run being copied
//    (16-byte cp.async, consecutive rows on different banks), the present group multiplied; one barrier per group;
//  * the runs are found from the table itself (smallest and largest entry of a warp's rows, merged to at most two windows):
//    any table is right.  Of a group whose rows do not fit the buffer every warp fetches its own, offset by offset;
//  * offsets that none of a warp's 16-row tiles has are skipped; a row without a neighbour reads a row of zeros;
//  * the order of sums is that of the tcgen05 kernels - offsets ascending, 32 bytes of a row per instruction, fp32 / int32
//    accumulators - and so are the results, bit for bit.
// Bound by instruction issue (about 100 instructions per 32 rows and offset, 16 of them products at 32 -> 32 channels), which
// is why the dense wide layers stay with tcgen05.  Measured on 300 k rows of 1.5 neighbours / 432 k rows of 6.5 (us):
//   16 -> 16 fp16  45 -> 32 / 66 -> 49 (tcgen05 before)     24 -> 40 fp16  332 -> 104 / 1758 -> 216 (row-walking kernel)
//   16 -> 32 int8  60 -> 41 / 244 -> 74 (pair kernel)       32 -> 32 fp16   63 -> 63 /   97 -> 107 (tcgen05: kept there)
#include "common.cuh"
#include "conv_strip.h"
#include "strip_common.cuh"

namespace sph {

namespace {

using namespace strip;

constexpr int kWarps = kStripThreads / 32;
constexpr int kGroup = 9;                 // offsets of a group: the 3 x 3 of one kernel height
constexpr int MT = 2;                     // 16-row tiles of a warp

__device__ __forceinline__ uint32_t pack16(float a, float b, int out_dtype) {
  if (out_dtype == SPH_F16) {
    const __half2 h = __floats2half2_rn(a, b);
    return *(const uint32_t*)&h;
  }
  const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  return *(const uint32_t*)&h;
}
__device__ __forceinline__ uint32_t sat8(float v) { return (uint32_t)(int)fminf(fmaxf(rintf(v), -127.f), 127.f) & 0xffu; }

// v[j] of lane t (of a quad) -> v[t] of lane j.
__device__ __forceinline__ void quad_transpose(uint32_t (&v)[4], int t) {
#pragma unroll
  for (int s = 1; s <= 2; s <<= 1) {
    const bool up = t & s;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if (j & s) continue;
      const uint32_t got = __shfl_xor_sync(0xffffffffu, up ? v[j] : v[j | s], s);
      if (up) v[j] = got; else v[j | s] = got;
    }
  }
}

// KS: 32-byte steps of a row, NT: 8-channel tiles of the output, WHOLE: rows are 32 * KS bytes.
template <int KS, int NT, bool WHOLE, int DT>
__global__ void __launch_bounds__(kStripThreads, (NT <= 4 && KS <= 2) ? 2 : 1) conv_strip_kernel(StripParams p) {
  after_previous<false>();
  extern __shared__ __align__(128) unsigned char smem[];
  constexpr int EPL = MT / 2;                              // table entries per lane and offset
  constexpr int WR = MT * 16;                              // rows of a warp
  constexpr int R = kWarps * WR;                           // rows of a tile
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int half = lane >> 4;                              // half of a 32-byte step this lane addresses for ldmatrix

  // [zero row][buffer 0][buffer 1][filter][runs]; positions inside are counted in 16-byte units from the zero row.  A row
  // takes an odd number of units, so that eight consecutive rows start on eight different groups of banks.
  const int rb16 = (p.row_bytes + 15) >> 4, pitch = rb16 | 1;
  const int buf_units = (p.cap * pitch + 7) & ~7;
  uint4* s_filter = (uint4*)(smem + (kZeroUnits + 2 * buf_units) * 16);
  int4* s_runs = (int4*)(s_filter + p.filter_units);       // [2][kWarps]
  const uint32_t smem0 = smem_u32(smem);
  const uint32_t operand0 = smem0 + half * 16;
  // rows that end inside a unit: the rest of it stays zero from here on
  const int zeros = WHOLE ? kZeroUnits : kZeroUnits + 2 * buf_units;
  for (int u = tid; u < zeros; u += kStripThreads) ((uint4*)smem)[u] = make_uint4(0u, 0u, 0u, 0u);
  for (int u = tid; u < p.filter_units; u += kStripThreads) cp_async_16(smem_u32(s_filter + u), p.filter + u, 16u);

  const int groups = (p.kv + kGroup - 1) / kGroup;
  const int my_tiles = (p.tiles - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;
  const int total = my_tiles * groups;
  const unsigned n_out = (unsigned)p.n_out;
  uint32_t bad = 0u;

  struct Place { int ti, g; };                             // tile (of this CTA) and group of a step
  auto after = [&](Place q) { return q.g + 1 < groups ? Place{q.ti, q.g + 1} : Place{q.ti + 1, 0}; };
  auto tile_row = [&](int ti) { return ((unsigned)blockIdx.x + (unsigned)ti * gridDim.x) * R + warp * WR; };

  int raw[kGroup][EPL];
  auto load_entries = [&](Place q) {
    const unsigned r = tile_row(q.ti) + lane;
    bool ok[EPL];
#pragma unroll
    for (int j = 0; j < EPL; ++j) ok[j] = q.ti < my_tiles && r + j * 32 < n_out;
    const int nk = p.kv - q.g * kGroup;
    const int64_t step = p.flip_k ? -p.n_out : p.n_out;
    const int* at = p.nbr + (int64_t)(p.flip_k ? p.kv - 1 - q.g * kGroup : q.g * kGroup) * p.n_out + r;
#pragma unroll
    for (int o = 0; o < kGroup; ++o) {
#pragma unroll
      for (int j = 0; j < EPL; ++j) raw[o][j] = (ok[j] && o < nk) ? __ldg(at + j * 32) : -1;
      at += step;
    }
  };
  // The warp's run of input rows, split in two where it is longer than half a buffer.
  auto post_run = [&](int slot) {
    unsigned lo = ~0u;
    int hi = -1, least = -1;
    auto run_of = [&]() {
      lo = ~0u; hi = -1; least = -1;
#pragma unroll
      for (int o = 0; o < kGroup; ++o)
#pragma unroll
        for (int j = 0; j < EPL; ++j) {
          lo = min(lo, (unsigned)raw[o][j]);
          hi = max(hi, raw[o][j]);
          least = min(least, raw[o][j]);
        }
      lo = __reduce_min_sync(0xffffffffu, lo);
      hi = __reduce_max_sync(0xffffffffu, hi);
    };
    run_of();
    if (hi >= (int)p.n_rows || __any_sync(0xffffffffu, least < -1)) {     // an entry that is neither a row nor -1
      bad = 1u;
#pragma unroll
      for (int o = 0; o < kGroup; ++o)
#pragma unroll
        for (int j = 0; j < EPL; ++j)
          if ((unsigned)raw[o][j] >= (unsigned)p.n_rows) raw[o][j] = -1;
      run_of();
    }
    int4 run = make_int4((int)min(lo, 0x7fffffffu), hi, INT_MAX, -1);
    if (hi >= 0 && hi - (int)lo >= p.cap / 2) {
      const int split = (int)lo + p.cap / 2;
      int hi1 = -1;
      unsigned lo2 = 0x7fffffffu;
#pragma unroll
      for (int o = 0; o < kGroup; ++o)
#pragma unroll
        for (int j = 0; j < EPL; ++j) {
          if (raw[o][j] < split) hi1 = max(hi1, raw[o][j]);
          else lo2 = min(lo2, (unsigned)raw[o][j]);
        }
      run = make_int4((int)lo, __reduce_max_sync(0xffffffffu, hi1), (int)__reduce_min_sync(0xffffffffu, lo2), hi);
    }
    if (lane == 0) s_runs[slot * kWarps + warp] = run;
  };
  auto stage = [&](const Windows& w, int slot) {
    if (!w.fit) return;
    const uint32_t dst = smem0 + (kZeroUnits + slot * buf_units) * 16;
    auto copy = [&](int base, int len, uint32_t to) {
      if (!WHOLE && (p.row_bytes & 15)) {
        copy_ragged_rows<kStripThreads>(p.rows, p.n_rows, base, len, p.row_bytes, pitch, to);
        return;
      }
      const unsigned n = len * rb16;
      const uint8_t* src = p.rows + (int64_t)base * p.row_bytes;
#pragma unroll 4
      for (unsigned u = tid; u < n; u += kStripThreads) {
        const unsigned at = WHOLE ? u + u / (KS * 2) : u + u / (unsigned)rb16 * (unsigned)(pitch - rb16);
        cp_async_16(to + at * 16, src + u * 16, 16u);
      }
    };
    copy(w.base1, w.len1, dst);
    if (w.len2) copy(w.base2, w.len2, dst + w.len1 * pitch * 16);
  };
  // A group's entries as positions in the buffer, two 16-bit ones to a register (0: the zero row), and whether enough of
  // them exist to multiply every 16-row tile at every offset.
  constexpr int NP = (kGroup * EPL + 1) / 2;
  struct Packed { uint32_t at[NP]; bool dense; };
  auto pack = [&](const Windows& w, int slot, Packed& out) {
    const int buf = kZeroUnits + slot * buf_units;
    const int off1 = buf - w.base1 * pitch, off2 = buf + (w.len1 - w.base2) * pitch, end1 = w.base1 + w.len1;
    const bool two = w.len2 > 0 && w.base2 > w.base1;      // windows in ascending order (else: compare both ends)
    int have = 0;
#pragma unroll
    for (int i = 0; i < NP; ++i) out.at[i] = 0u;
#pragma unroll
    for (int o = 0; o < kGroup; ++o)
#pragma unroll
      for (int j = 0; j < EPL; ++j) {
        const int e = raw[o][j], i = o * EPL + j;
        int off = off1;
        if (w.len2 > 0) off = (two ? e < end1 : (e >= w.base1 && e < end1)) ? off1 : off2;
        const uint32_t at = e >= 0 ? (uint32_t)(e * pitch + off) : 0u;
        have += e >= 0;
        out.at[i / 2] |= i & 1 ? at << 16 : at;
      }
    // below 3 rows in 16 on average the tiles without any are worth skipping
    out.dense = __reduce_add_sync(0xffffffffu, have) * 16 >= kGroup * WR * 3;
  };

  uint32_t acc[MT][NT][4];
  // One offset: `a(m, s, frag)` loads the operand of 16-row tile m, step s.
  auto multiply = [&](int k, uint32_t tiles, auto&& a) {
    const uint4* w = s_filter + k * (KS * (NT / 2) * 32) + lane;
#pragma unroll
    for (int s = 0; s < KS; ++s) {
      uint4 b[NT / 2];
#pragma unroll
      for (int n = 0; n < NT / 2; ++n) b[n] = w[(s * (NT / 2) + n) * 32];
#pragma unroll
      for (int m = 0; m < MT; ++m) {
        if (tiles >> m & 1u) {                               // uniform
          uint32_t f[4];
          a(m, s, f);
#pragma unroll
          for (int n = 0; n < NT / 2; ++n) {
            mma_step<DT>(acc[m][2 * n], f, b[n].x, b[n].y);
            mma_step<DT>(acc[m][2 * n + 1], f, b[n].z, b[n].w);
          }
        }
      }
    }
  };

  Packed cur, nxt;
  Windows wn;
  bool cur_fit;
  Place here{0, 0}, there = after(here);
  load_entries(here);
  post_run(0);
  __syncthreads();
  wn = merge_runs<kWarps>(s_runs, p.cap);
  stage(wn, 0);
  pack(wn, 0, cur);
  cur_fit = wn.fit;
  load_entries(there);
  post_run(1);
  cp_async_wait_all();
  __syncthreads();

  for (int j = 0; j < total; ++j) {
    // the next group's rows start moving, the entries of the one behind it are requested
    wn = merge_runs<kWarps>(s_runs + ((j + 1) & 1) * kWarps, p.cap);
    stage(wn, (j + 1) & 1);
    pack(wn, (j + 1) & 1, nxt);
    const Place behind = after(there);
    load_entries(behind);

    if (here.g == 0) {
#pragma unroll
      for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int n = 0; n < NT; ++n)
#pragma unroll
          for (int q = 0; q < 4; ++q) acc[m][n][q] = 0u;
    }
    const int k0 = here.g * kGroup;
    // addresses of the pieces this lane fetches for ldmatrix: row lane % 16 of every tile at offset o
    auto operands = [&](int o, uint32_t (&at)[MT]) {
#pragma unroll
      for (int j = 0; j < EPL; ++j) {
        const int i = o * EPL + j;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const uint32_t x = __shfl_sync(0xffffffffu, cur.at[i / 2], 16 * h + (lane & 15));
          at[2 * j + h] = operand0 + (i & 1 ? x >> 16 : x & 0xffffu) * 16u;
        }
      }
    };
    auto fetch = [&](uint32_t at, int s, uint32_t (&f)[4]) {
      // one instruction for the whole warp: a half-warp whose piece lies beyond the row points at the zero row
      ldmatrix4(f, WHOLE || 2 * s + half < rb16 ? at + s * 32 : smem0);
    };
    if (cur_fit && cur.dense && k0 + kGroup <= p.kv) {
      // most tiles have a neighbour at most offsets: all of them are multiplied (rows of zeros change nothing), without
      // branches between the loads of one offset and the products of another
#pragma unroll
      for (int o = 0; o < kGroup; ++o) {
        uint32_t at[MT];
        operands(o, at);
        const uint4* w = s_filter + (k0 + o) * (KS * (NT / 2) * 32) + lane;
#pragma unroll
        for (int s = 0; s < KS; ++s) {
          uint32_t f[MT][4];
#pragma unroll
          for (int m = 0; m < MT; ++m) fetch(at[m], s, f[m]);
#pragma unroll
          for (int n = 0; n < NT / 2; ++n) {
            const uint4 b = w[(s * (NT / 2) + n) * 32];
#pragma unroll
            for (int m = 0; m < MT; ++m) {
              mma_step<DT>(acc[m][2 * n], f[m], b.x, b.y);
              mma_step<DT>(acc[m][2 * n + 1], f[m], b.z, b.w);
            }
          }
        }
      }
    } else if (cur_fit) {
#pragma unroll
      for (int o = 0; o < kGroup; ++o) {
        uint32_t at[MT];
        operands(o, at);
        uint32_t tiles = 0u;
#pragma unroll
        for (int m = 0; m < MT; ++m) tiles |= (__any_sync(0xffffffffu, at[m] != operand0) ? 1u : 0u) << m;
        if (tiles) multiply(k0 + o, tiles, [&](int m, int s, uint32_t (&f)[4]) { fetch(at[m], s, f); });
      }
    } else {
      // The rows of this group are too far apart for a buffer (filters whose nine offsets span several lines of columns, input
      // gradients of strided layers): every warp fetches the rows of its own 32 into its share of the buffer the group does not
      // use, up to three offsets at a time, the next ones' entries in flight with them.  (Fragments straight from global memory,
      // four bytes a load and one offset behind the other: 3 x 3 x 1 16 -> 16 on 547 k rows 88 -> 62 us, 5 -> 7 131 -> 88; the 16-channel
      // gradient of a strided layer 99 -> 61.)
      const int share = p.cap / kWarps, held = min(share / WR, 3);           // rows; at least 320 / 8
      const int mine = kZeroUnits + (j & 1) * buf_units + warp * share * pitch;
      const unsigned r = tile_row(here.ti) + lane;
      const int nk = min(kGroup, p.kv - k0);
      int e[3];
      auto entries = [&](int o0) {
#pragma unroll
        for (int q = 0; q < 3; ++q) {
          const int k = k0 + o0 + q;
          e[q] = q < held && o0 + q < nk && r < n_out ? __ldg(p.nbr + (int64_t)(p.flip_k ? p.kv - 1 - k : k) * p.n_out + r) : -1;
          if ((unsigned)e[q] >= (unsigned)p.n_rows) e[q] = -1;
        }
      };
      entries(0);
      for (int o0 = 0; o0 < nk; o0 += held) {
        uint32_t have[3];
#pragma unroll
        for (int q = 0; q < 3; ++q) {
          have[q] = __ballot_sync(0xffffffffu, e[q] >= 0);
          if (e[q] >= 0) {
            const uint8_t* src = p.rows + (int64_t)e[q] * p.row_bytes;
            const uint32_t dst = smem0 + (mine + (q * WR + lane) * pitch) * 16;
            if (WHOLE) {
#pragma unroll
              for (int u = 0; u < 2 * KS; ++u) cp_async_16(dst + u * 16, src + u * 16, 16u);
            } else {
              copy_ragged_row(src, p.row_bytes, dst);
            }
          }
        }
        entries(o0 + held);
        cp_async_wait_all();
        __syncwarp();
#pragma unroll
        for (int q = 0; q < 3; ++q) {
          if (have[q] == 0u) continue;
          uint32_t at[MT];
#pragma unroll
          for (int m = 0; m < MT; ++m) {
            const int row = 16 * m + (lane & 15);
            at[m] = operand0 + (have[q] >> row & 1u ? (uint32_t)(mine + (q * WR + row) * pitch) * 16u : 0u);
          }
          const uint32_t tiles = ((have[q] & 0xffffu) ? 1u : 0u) | ((have[q] >> 16) ? 2u : 0u);
          multiply(k0 + o0 + q, tiles, [&](int m, int s, uint32_t (&f)[4]) { fetch(at[m], s, f); });
        }
        __syncwarp();
      }
    }

    if (here.g == groups - 1) {
      // ---- epilogue: the lane holds channels 8n + 2t, + 1 of rows g and g + 8 of every 16-row tile
      const int g = lane >> 2, t = lane & 3;
      const int64_t row0 = tile_row(here.ti);
      constexpr int G = NT % 4 == 0 ? 4 : 2;              // channel tiles of a store
#pragma unroll
      for (int nn = 0; nn < NT; nn += G) {
        if (nn * 8 >= p.N) break;
        float sc[G][2], bi[G][2];
#pragma unroll
        for (int i = 0; i < G; ++i)
#pragma unroll
          for (int q = 0; q < 2; ++q) {
            const int c = (nn + i) * 8 + 2 * t + q;
            sc[i][q] = (p.scale && c < p.N) ? __ldg(p.scale + c) : 1.f;
            bi[i][q] = c < p.N ? p.bias.at<DT != SPH_I8>(c) : 0.f;
          }
#pragma unroll
        for (int m = 0; m < MT; ++m)
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const int64_t r = row0 + m * 16 + h * 8 + g;
            float v[G][2];
#pragma unroll
            for (int i = 0; i < G; ++i)
#pragma unroll
              for (int q = 0; q < 2; ++q) {
                const uint32_t x = acc[m][nn + i][h * 2 + q];
                const float y = fmaf(DT == SPH_I8 ? (float)(int)x : __uint_as_float(x), sc[i][q], bi[i][q]);
                v[i][q] = p.relu ? fmaxf(y, 0.f) : y;
              }
            if (G == 4 && (nn + 4) * 8 <= p.N && p.N % 8 == 0) {
              // lane t gets the 8 channels of tile nn + t: one vector store per row and lane
              uint32_t w[4];
              const int64_t at = r * p.N + (nn + t) * 8;
              if (p.out_dtype == SPH_F16 || p.out_dtype == SPH_BF16) {
#pragma unroll
                for (int i = 0; i < 4; ++i) w[i] = pack16(v[i % G][0], v[i % G][1], p.out_dtype);
                quad_transpose(w, t);
                if (r < p.n_out) *(uint4*)((uint16_t*)p.out + at) = make_uint4(w[0], w[1], w[2], w[3]);
              } else if (p.out_dtype == SPH_I8) {
#pragma unroll
                for (int i = 0; i < 4; ++i) w[i] = sat8(v[i % G][0]) | sat8(v[i % G][1]) << 8;
                quad_transpose(w, t);
                if (r < p.n_out) *(uint2*)((uint8_t*)p.out + at) = make_uint2(w[0] | w[1] << 16, w[2] | w[3] << 16);
              } else {
                uint32_t u[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                  w[i] = __float_as_uint(v[i % G][0]);
                  u[i] = __float_as_uint(v[i % G][1]);
                }
                quad_transpose(w, t);
                quad_transpose(u, t);
                if (r < p.n_out) {
                  ((uint4*)((float*)p.out + at))[0] = make_uint4(w[0], u[0], w[1], u[1]);
                  ((uint4*)((float*)p.out + at))[1] = make_uint4(w[2], u[2], w[3], u[3]);
                }
              }
            } else if (r < p.n_out) {
#pragma unroll
              for (int i = 0; i < G; ++i) {
                const int c = (nn + i) * 8 + 2 * t;
                const int64_t at = r * p.N + c;
                if (p.N % 2 == 0) {
                  if (c >= p.N) continue;
                  if (p.out_dtype == SPH_F32) *(float2*)((float*)p.out + at) = make_float2(v[i][0], v[i][1]);
                  else if (p.out_dtype == SPH_I8) *(uint16_t*)((uint8_t*)p.out + at) = (uint16_t)(sat8(v[i][0]) | sat8(v[i][1]) << 8);
                  else *(uint32_t*)((uint16_t*)p.out + at) = pack16(v[i][0], v[i][1], p.out_dtype);
                } else {
#pragma unroll
                  for (int q = 0; q < 2; ++q) {
                    if (c + q >= p.N) continue;
                    if (p.out_dtype == SPH_F32) ((float*)p.out)[at + q] = v[i][q];
                    else if (p.out_dtype == SPH_I8) ((uint8_t*)p.out)[at + q] = (uint8_t)sat8(v[i][q]);
                    else ((uint16_t*)p.out)[at + q] = (uint16_t)pack16(v[i][q], v[i][q], p.out_dtype);
                  }
                }
              }
            }
          }
      }
    }
    post_run(j & 1);
    cp_async_wait_all();
    __syncthreads();
    cur = nxt;
    cur_fit = wn.fit;
    here = there;
    there = behind;
  }
  if (bad && p.status) atomicOr(p.status, SPH_STATUS_BAD_INDEX);
}

template <int KS, int NT, bool WHOLE, int DT>
int launch_strip_kernel(StripParams& p, cudaStream_t st) {
  constexpr int R = kWarps * MT * 16;
  p.tiles = (int)div_up64(p.n_out, R);
  const int pitch = ((p.row_bytes + 15) / 16 | 1) * 16;
  auto kern = conv_strip_kernel<KS, NT, WHOLE, DT>;
  // a buffer holds 3 input rows per output row where there is room (columns at the edges of a tile included), and two CTAs
  // share an SM where the registers let them
  const int ctas = (NT <= 4 && KS <= 2) ? 2 : 1;
  const int fixed = strip_fixed_bytes(p.filter_units);
  int cap = (kStripSmem / ctas - fixed) / (2 * pitch);
  int per_sm = ctas;
  if (cap < R + 64) {
    cap = (kStripSmem - fixed) / (2 * pitch);
    per_sm = 1;
  }
  p.cap = cap < 3 * R ? cap : 3 * R;
  const int smem = fixed + 2 * ((p.cap * (pitch / 16) + 7) & ~7) * 16;
  SPH_CUDA(allow_smem(kern, kStripSmem));
  const int sms = current_sm_count();
  if (sms <= 0) return SPH_ERR_CUDA;
  const int grid = p.tiles < sms * per_sm ? p.tiles : sms * per_sm;
  launch(kern, grid, kStripThreads, smem, st, p);
  SPH_LAUNCH_CHECK();
  return SPH_OK;
}

template <int DT>
int launch_strip(StripParams& p, const StripShape& s, cudaStream_t st) {
#define SPH_STRIP(KS, NT)                                                                                  \
  if (s.ks == KS && s.nt == NT)                                                                            \
    return s.whole ? launch_strip_kernel<KS, NT, true, DT>(p, st) : launch_strip_kernel<KS, NT, false, DT>(p, st)
  SPH_STRIP(1, 2); SPH_STRIP(1, 4); SPH_STRIP(1, 8);
  SPH_STRIP(2, 2); SPH_STRIP(2, 4); SPH_STRIP(2, 8);
  SPH_STRIP(4, 2); SPH_STRIP(4, 4); SPH_STRIP(4, 8);
#undef SPH_STRIP
  set_error("conv_strip: no kernel for this shape");
  return SPH_ERR_UNSUPPORTED;
}

}  // namespace

}  // namespace sph
