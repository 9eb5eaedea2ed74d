// Weight gradient over the present pairs (mma.sync + ldmatrix): fp16 / bf16 layers of up to 64 channels on either side.
//
//   dW[k] (K x N) += sum over the pairs (i, o) of offset k of  X[i,:]^T dY[o,:]
//
// The sum runs over rows, so only rows that form a pair need to be multiplied - 1.2 to 22 of 27 slots of a LiDAR level's
// table.  A tcgen05 kernel has to walk every slot: its operand is a tile of 256 gathered rows, absent ones as zeros, and each
// of them crosses shared memory.  Here the pairs of an offset are compacted into a list, and ldmatrix (transposing) picks
// both operands of 16 pairs out of staged rows: the run of input rows that a tile of 256 output rows has at the 9 offsets
// of one kernel height (see conv_strip.cuh), and the dY rows of the tile themselves.
//
//  * a CTA serves one group of 9 offsets, one offset per warp, and walks tiles of output rows: table entries of the tile
//    after next in flight, the next tile's rows being copied, the present tile multiplied; one barrier per tile;
//  * the centre offset of a submanifold layer has a pair for every row, the others for a fifth: three more warps (nine warps
//    leave room for twelve) take three quarters of the longest list, found on the CTA's first tile;
//  * of a tile whose input rows lie too far apart for a buffer every warp fetches those of its own pairs;
//  * more than 32 input channels are two launches' worth of CTAs, 32 channels each: the accumulators of 64 x 64 would spill;
//  * a warp keeps its K x N gradient in registers over all its tiles and adds it to the fp32 gradient once, at the end (the
//    reference writes [NTile,KV,iC,oC] partials and sums them, src/sphconv/rule_conv.cu:483-484,517).
// Measured (us, tcgen05 kernel -> this one): 432 k rows of 6.5 pairs 16 -> 16 80 -> 68, 32 -> 32 159 -> 102, 64 -> 64 287 -> 241;
// a strided layer's 343 k rows of 4.2 pairs 32 -> 64 194 -> 96; 24 -> 40 1183 -> 132 (row-walking kernel).
#include "strip_common.cuh"

namespace sph {

namespace {

using namespace strip;

constexpr int kGroup = 9;                 // offsets of a CTA, one per warp
constexpr int kHelpers = 3;               // warps that share the longest of the nine lists with its owner
constexpr int kThreads = (kGroup + kHelpers) * 32;
constexpr int kRows = 256;                // output rows of a tile
constexpr int kChunks = kRows / 32;
constexpr int kSmem = 222 * 1024;

struct WgradStripParams {
  const uint8_t* rows;                    // X [n_rows, K]
  const uint8_t* dout;                    // dY [n_out, N]
  const int* nbr;                         // [KV, n_out]
  float* dw;                              // [KV, K, N], accumulated into
  int64_t n_rows, n_out;
  int kv, K, N;
  int groups, halves, slices, tiles;       // halves: parts of 32 input channels
  int cap;                                // input rows a buffer holds
  int x_piece;                            // bytes of a row of X that may be copied at a time
  int pairs_of_floats;                    // the gradient may be added to two floats at a time
  int* status;
};

// Channels [c0, c0 + n) of consecutive 16-bit rows -> rows `pitch` units apart.
__device__ __forceinline__ void copy_rows(const uint8_t* tensor, int64_t n_rows, int base, int len, int channels, int c0, int n_ch,
                                          int pitch, uint32_t to) {
  if (channels & 1) {
    copy_odd_rows<kThreads>((const uint16_t*)tensor, n_rows * channels, base, len, channels, c0, n_ch, pitch, to);
    return;
  }
  const uint8_t* rows = tensor + c0 * 2;
  const int row_bytes = channels * 2, bytes = n_ch * 2;
  const uint8_t* src = rows + (int64_t)base * row_bytes;
  if (((uintptr_t)rows | row_bytes | bytes) & 15) {         // 8- or 4-byte pieces
    const int piece = (((uintptr_t)rows | row_bytes | bytes) & 7) ? 4 : 8;
    const unsigned per = bytes / piece, n = per * len;
    for (unsigned u = threadIdx.x; u < n; u += kThreads) {
      const unsigned r = u / per, at = u % per * piece;
      if (piece == 8) cp_async_8(to + r * pitch * 16 + at, src + (size_t)r * row_bytes + at);
      else cp_async_4(to + r * pitch * 16 + at, src + (size_t)r * row_bytes + at);
    }
    return;
  }
  const unsigned per = (unsigned)bytes >> 4, n = per * len;
  const bool pow2 = (per & (per - 1)) == 0;
  const int sh = __ffs(per) - 1;
#pragma unroll 4
  for (unsigned u = threadIdx.x; u < n; u += kThreads) {
    const unsigned r = pow2 ? u >> sh : u / per, c = u - r * per;
    cp_async_16(to + (r * pitch + c) * 16, src + (size_t)r * row_bytes + c * 16, 16u);
  }
}

// n channels of one row by one thread; piece: bytes at a time (16, 8, 4 or 2).
__device__ __forceinline__ void copy_channels(const uint16_t* src, int n, int piece, uint32_t to) {
  const int bytes = n * 2;
  if (piece == 16) {
    for (int b = 0; b < bytes; b += 16) cp_async_16(to + b, (const uint8_t*)src + b, 16u);
  } else if (piece == 8) {
    for (int b = 0; b < bytes; b += 8) cp_async_8(to + b, (const uint8_t*)src + b);
  } else if (piece == 4) {
    for (int b = 0; b < bytes; b += 4) cp_async_4(to + b, (const uint8_t*)src + b);
  } else {
#pragma unroll 4
    for (int c = 0; c < n; ++c) asm volatile("st.shared.u16 [%0], %1;" ::"r"(to + c * 2), "h"(__ldg(src + c)) : "memory");
  }
}

// KT: tiles of 16 input channels, NP: pairs of 8-channel tiles of the output.
template <int KT, int NP, int DT>
__global__ void __launch_bounds__(kThreads, KT * NP <= 2 ? 2 : 1) conv_wgrad_strip_kernel(WgradStripParams p) {
  after_previous<false>();
  extern __shared__ __align__(128) unsigned char smem[];
  constexpr int PX = 2 * KT + 1, PY = 2 * NP + 1;          // 16-byte units between rows (odd: other banks)
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int x_units = (p.cap * PX + 7) & ~7;
  constexpr int y_units = (kRows * PY + 7) & ~7;
  const int x0 = kZeroUnits, y0 = x0 + 2 * x_units;        // positions in 16-byte units
  uint32_t* s_lists = (uint32_t*)(smem + (y0 + 2 * y_units) * 16);      // [kGroup][2][kRows]
  const bool owner = warp < kGroup;
  int4* s_runs = (int4*)(smem + (y0 + 2 * y_units) * 16 + kGroup * 2 * kRows * 4);
  int* s_count = (int*)(s_runs + 2 * kGroup);              // [2][kGroup] pairs per offset
  const uint32_t smem0 = smem_u32(smem);
  // the zero row, and what lies between a row's end and the next row (channels beyond K and N)
  for (int u = tid; u < y0 + 2 * y_units; u += kThreads) ((uint4*)smem)[u] = make_uint4(0u, 0u, 0u, 0u);

  const int part_of = (int)blockIdx.x % (p.groups * p.halves), slice = (int)blockIdx.x / (p.groups * p.halves);
  const int group = part_of % p.groups, ch0 = part_of / p.groups * 32;     // first input channel
  const int kc = min(KT * 16, p.K - ch0);
  int k = owner ? group * kGroup + warp : p.kv;            // a helper learns its offset from the first tile
  const int my_tiles = slice < p.tiles ? (p.tiles - slice + p.slices - 1) / p.slices : 0;
  auto first_row = [&](int ti) { return ((int64_t)slice + (int64_t)ti * p.slices) * kRows; };
  const int* plane = p.nbr + (int64_t)(owner ? k : 0) * p.n_out;
  const unsigned lower = (1u << lane) - 1u;
  const int share = p.cap / (kThreads / 32);               // rows of a buffer per warp: 32 at least
  bool bad = false;

  int e[kChunks];
  auto load_entries = [&](int ti) {
    const int64_t r = first_row(ti) + lane;
#pragma unroll
    for (int h = 0; h < kChunks; ++h)
      e[h] = (ti < my_tiles && owner && k < p.kv && r + h * 32 < p.n_out) ? __ldg(plane + r + h * 32) : -1;
  };
  // The warp's run of input rows, split in two where it is longer than half a buffer.
  auto post_run = [&](int slot) {
    unsigned lo = ~0u;
    int hi = -1;
#pragma unroll
    for (int h = 0; h < kChunks; ++h) {
      if ((unsigned)e[h] >= (unsigned)p.n_rows) {
        bad |= e[h] != -1;                                 // neither a row nor -1
        e[h] = -1;
      }
      lo = min(lo, (unsigned)e[h]);
      hi = max(hi, e[h]);
    }
    lo = __reduce_min_sync(0xffffffffu, lo);
    hi = __reduce_max_sync(0xffffffffu, hi);
    int4 run = make_int4((int)min(lo, 0x7fffffffu), hi, INT_MAX, -1);
    if (hi >= 0 && hi - (int)lo >= p.cap / 2) {
      const int split = (int)lo + p.cap / 2;
      int hi1 = -1;
      unsigned lo2 = 0x7fffffffu;
#pragma unroll
      for (int h = 0; h < kChunks; ++h) {
        if (e[h] < split) hi1 = max(hi1, e[h]);
        else lo2 = min(lo2, (unsigned)e[h]);
      }
      run = make_int4((int)lo, __reduce_max_sync(0xffffffffu, hi1), (int)__reduce_min_sync(0xffffffffu, lo2), hi);
    }
    if (lane == 0 && owner) s_runs[slot * kGroup + warp] = run;
  };
  auto stage = [&](const Windows& w, int ti, int slot) {
    const int64_t r = first_row(ti);
    const int n = ti < my_tiles ? (int)min((int64_t)kRows, p.n_out - r) : 0;
    copy_rows(p.dout, p.n_out, (int)r, n, p.N, 0, p.N, PY, smem0 + (y0 + slot * y_units) * 16);
    if (!w.fit) return;
    const uint32_t to = smem0 + (x0 + slot * x_units) * 16;
    copy_rows(p.rows, p.n_rows, w.base1, w.len1, p.K, ch0, kc, PX, to);
    if (w.len2) copy_rows(p.rows, p.n_rows, w.base2, w.len2, p.K, ch0, kc, PX, to + w.len1 * PX * 16);
  };
  // The warp's pairs of a tile: position of the input row | position of the dY row << 16, padded to a multiple of 16 with
  // pairs of zero rows.  Where the input rows are not staged: 1 + the pair's row in the tile instead of the former.
  auto list_pairs = [&](const Windows& w, int slot) {
    if (!owner) return;
    uint32_t* list = s_lists + (warp * 2 + slot) * kRows;
    const int xs = x0 + slot * x_units, ys = y0 + slot * y_units;
    int n = 0;
#pragma unroll
    for (int h = 0; h < kChunks; ++h) {
      const uint32_t m = __ballot_sync(0xffffffffu, e[h] >= 0);
      if (e[h] >= 0) {
        const int r = (unsigned)(e[h] - w.base1) < (unsigned)w.len1 ? e[h] - w.base1 : w.len1 + e[h] - w.base2;
        const int row = h * 32 + lane;
        list[n + __popc(m & lower)] = (uint32_t)(w.fit ? xs + r * PX : 1 + row) | (uint32_t)(ys + row * PY) << 16;
      }
      n += __popc(m);
    }
    if (lane < (-n & 15)) list[n + lane] = 0u;
    if (lane == 0) s_count[slot * kGroup + warp] = n;
  };

  float acc_f[KT][NP * 2][4];
  uint32_t (*acc)[NP * 2][4] = (uint32_t (*)[NP * 2][4])acc_f;
#pragma unroll
  for (int m = 0; m < KT; ++m)
#pragma unroll
    for (int n = 0; n < NP * 2; ++n)
#pragma unroll
      for (int q = 0; q < 4; ++q) acc_f[m][n][q] = 0.f;

  // pair and 8-channel half that this lane addresses in either operand's four matrices
  const int a_pair = (lane & 7) + (lane >> 4) * 8, b_pair = (lane & 7) + (lane >> 3 & 1) * 8;
  const uint32_t a_base = smem0 + (lane >> 3 & 1) * 16, b_base = smem0 + (lane >> 4) * 16;

  load_entries(0);
  post_run(0);
  __syncthreads();
  Windows wn = merge_runs<kGroup>(s_runs, p.cap);
  stage(wn, 0, 0);
  list_pairs(wn, 0);
  bool fit = wn.fit;
  load_entries(1);
  post_run(1);
  cp_async_wait_all();
  __syncthreads();

  int longest = 0;
  for (int w = 1; w < kGroup; ++w)
    if (s_count[w] > s_count[longest]) longest = w;
  const int list_of = owner ? warp : longest;              // whose list this warp works on, its first chunk and step
  const int part = owner ? 0 : warp - kGroup + 1, parts = list_of == longest ? kHelpers + 1 : 1;
  k = group * kGroup + list_of;

  for (int ti = 0; ti < my_tiles; ++ti) {
    const int slot = ti & 1, other = slot ^ 1;
    wn = merge_runs<kGroup>(s_runs + other * kGroup, p.cap);
    stage(wn, ti + 1, other);
    list_pairs(wn, other);
    load_entries(ti + 2);

    const uint32_t* list = s_lists + (list_of * 2 + slot) * kRows;
    const int n = s_count[slot * kGroup + list_of];
    auto products = [&](const uint32_t (&a)[KT][4], uint32_t b_at) {          // 16 pairs
#pragma unroll
      for (int j = 0; j < NP; ++j) {
        uint32_t b[4];
        ldmatrix4_trans(b, b_at + j * 32);
#pragma unroll
        for (int m = 0; m < KT; ++m) {
          mma_step<DT>(acc[m][2 * j], a[m], b[0], b[1]);
          mma_step<DT>(acc[m][2 * j + 1], a[m], b[2], b[3]);
        }
      }
    };
    if (fit) {
#pragma unroll 1
      for (int c = part * 16; c < n; c += parts * 16) {
        const uint32_t ea = list[c + a_pair], eb = list[c + b_pair];
        const uint32_t b_at = b_base + (eb >> 16) * 16, a_at = a_base + (ea & 0xffffu) * 16;
        uint32_t a[KT][4];
#pragma unroll
        for (int m = 0; m < KT; ++m) ldmatrix4_trans(a[m], a_at + m * 32);
        products(a, b_at);
      }
    } else {
      // The input rows of this tile are too far apart for a buffer: every warp fetches those of its pairs into its share of the
      // one the tile does not use, two steps at a time.  (Fragments straight from global memory, an element a load: 3 x 3 x 1
      // 32 -> 32 on 531 k rows 187 -> 107 us.)
      const int mine = x0 + slot * x_units + warp * share * PX;
#pragma unroll 1
      for (int c = part * 32; c < n; c += parts * 32) {
        const int idx = c + lane < n ? (int)(list[c + lane] & 0xffffu) - 1 : -1;
        int row = idx < 0 ? -1 : __ldg(p.nbr + (int64_t)k * p.n_out + first_row(ti) + idx);
        if ((unsigned)row >= (unsigned)p.n_rows) row = -1;
        const uint32_t have = __ballot_sync(0xffffffffu, row >= 0);
        if (row >= 0)
          copy_channels((const uint16_t*)p.rows + (int64_t)row * p.K + ch0, kc, p.x_piece, smem0 + (mine + lane * PX) * 16);
        cp_async_wait_all();
        __syncwarp();
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          if (c + h * 16 >= n) break;
          const int i = h * 16 + a_pair;
          const uint32_t a_at = a_base + (have >> i & 1u ? (uint32_t)(mine + i * PX) * 16u : 0u);
          uint32_t a[KT][4];
#pragma unroll
          for (int m = 0; m < KT; ++m) ldmatrix4_trans(a[m], a_at + m * 32);
          products(a, b_base + (list[c + h * 16 + b_pair] >> 16) * 16);
        }
        __syncwarp();
      }
    }
    post_run(slot);
    cp_async_wait_all();
    __syncthreads();
    fit = wn.fit;
  }

  if (k < p.kv && my_tiles > 0) {
    float* dw = p.dw + ((int64_t)k * p.K + ch0) * p.N;
#pragma unroll
    for (int m = 0; m < KT; ++m)
#pragma unroll
      for (int j = 0; j < NP * 2; ++j)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int ch = m * 16 + h * 8 + (lane >> 2), c = j * 8 + (lane & 3) * 2;
          if (ch >= kc || c >= p.N) continue;
          float* at = dw + ch * p.N + c;
          if (p.pairs_of_floats) {
            atomicAdd((float2*)at, make_float2(acc_f[m][j][2 * h], acc_f[m][j][2 * h + 1]));
          } else {
            atomicAdd(at, acc_f[m][j][2 * h]);
            if (c + 1 < p.N) atomicAdd(at + 1, acc_f[m][j][2 * h + 1]);
          }
        }
  }
  if (bad && p.status) atomicOr(p.status, SPH_STATUS_BAD_INDEX);
}

int fixed_bytes(int np) {
  return (kZeroUnits + 2 * ((kRows * (2 * np + 1) + 7) & ~7)) * 16 + kGroup * 2 * kRows * 4 + 2 * kGroup * 20;
}

template <int KT, int NP, int DT>
int launch_wgrad_strip(WgradStripParams& p, cudaStream_t st) {
  constexpr int PX = 2 * KT + 1;
  auto kern = conv_wgrad_strip_kernel<KT, NP, DT>;
  // three input rows per output row where there is room; two CTAs on an SM where their buffers still hold a tile's rows
  int per_sm = KT * NP <= 2 ? 2 : 1;
  int cap = (kSmem / per_sm - fixed_bytes(NP)) / (2 * PX * 16);
  if (cap < 2 * kRows && per_sm == 2) {
    per_sm = 1;
    cap = (kSmem - fixed_bytes(NP)) / (2 * PX * 16);
  }
  p.cap = (cap < 3 * kRows ? cap : 3 * kRows) & ~7;
  static_assert((kSmem - (kZeroUnits + 2 * ((kRows * (2 * 4 + 1) + 7) & ~7)) * 16 - kGroup * 2 * kRows * 4 - 2 * kGroup * 20) /
                        (2 * 5 * 16) >= 32 * (kThreads / 32), "a warp's share of a buffer holds the rows of two steps");
  const int smem = fixed_bytes(NP) + 2 * ((p.cap * PX + 7) & ~7) * 16;
  SPH_CUDA(allow_smem(kern, kSmem));
  const int sms = current_sm_count();
  if (sms <= 0) return SPH_ERR_CUDA;
  int slices = sms * per_sm / (p.groups * p.halves);
  if (slices > p.tiles) slices = p.tiles;
  p.slices = slices < 1 ? 1 : slices;
  launch(kern, p.slices * p.groups * p.halves, kThreads, smem, st, p);
  SPH_LAUNCH_CHECK();
  return SPH_OK;
}

template <int DT>
int launch_wgrad_shape(WgradStripParams& p, int kt, int np, cudaStream_t st) {
#define SPH_WG(KT, NP) if (kt == KT && np == NP) return launch_wgrad_strip<KT, NP, DT>(p, st)
  SPH_WG(1, 1); SPH_WG(1, 2); SPH_WG(1, 4);
  SPH_WG(2, 1); SPH_WG(2, 2); SPH_WG(2, 4);
#undef SPH_WG
  return SPH_ERR_UNSUPPORTED;
}

}  // namespace


bool conv_wgrad_strip_supported(int dtype, int K, int N) {
  return (dtype == SPH_F16 || dtype == SPH_BF16) && K >= 1 && N >= 1 && K <= 64 && N <= 64;
}

int conv_wgrad_strip(const void* rows, const void* dout, int dtype, int64_t n_rows, const int* nbr, int64_t n_out, int kv,
                     int K, int N, float* dw, int* status, cudaStream_t st) {
  if (!conv_wgrad_strip_supported(dtype, K, N)) {
    set_error("conv_wgrad_strip: unsupported dtype/shape");
    return SPH_ERR_UNSUPPORTED;
  }
  WgradStripParams p;
  p.rows = (const uint8_t*)rows; p.dout = (const uint8_t*)dout; p.nbr = nbr; p.dw = dw;
  p.n_rows = n_rows; p.n_out = n_out;
  p.kv = kv; p.K = K; p.N = N; p.status = status;
  p.groups = div_up(kv, kGroup);
  p.halves = div_up(K, 32);
  p.tiles = (int)div_up64(n_out, kRows);
  // rows, and the halves of them that start 32 channels in, as wide as their addresses and lengths allow (K odd: single elements)
  const uintptr_t at = (uintptr_t)rows | (uintptr_t)(K * 2);
  p.x_piece = at & 2 ? 2 : at & 4 ? 4 : at & 8 ? 8 : 16;
  p.pairs_of_floats = N % 2 == 0 && ((uintptr_t)dw & 7u) == 0;
  const int kt = K <= 16 ? 1 : 2, np = N <= 16 ? 1 : N <= 32 ? 2 : 4;
  return dtype == SPH_F16 ? launch_wgrad_shape<SPH_F16>(p, kt, np, st) : launch_wgrad_shape<SPH_BF16>(p, kt, np, st);
}

}  // namespace sph
