// fp32 arithmetic (FFMA) kernels of the rule-driven convolution: float32 rows (the 1e-4 tolerance rules out single-pass
// TF32) and 16-bit rows of channel counts the tensor-core kernels do not take.
//
// Both kernels work on the PRESENT pairs only - the FMA pipe is what bounds a float32 layer, so a slot without a
// neighbour must cost nothing - and both are register-blocked outer products over rows staged in shared memory.
#include "common.cuh"
#include "tc_common.cuh"

namespace sph {

namespace {

using tc::cp_async_16;
using tc::cp_async_commit;
using tc::cp_async_wait_pending;
using tc::smem_u32;

// One element global -> shared as a float; float32 elements asynchronously.
__device__ __forceinline__ void stage_one(float* dst, const float* src, bool ok) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(ok ? 4u : 0u));
}
__device__ __forceinline__ void stage_one(float* dst, const __half* src, bool ok) { *dst = ok ? __half2float(*src) : 0.f; }
__device__ __forceinline__ void stage_one(float* dst, const __nv_bfloat16* src, bool ok) { *dst = ok ? __bfloat162float(*src) : 0.f; }

__device__ __forceinline__ void store_one(void* out, int out_dtype, int64_t idx, float v) {
  switch (out_dtype) {
    case SPH_F32: ((float*)out)[idx] = v; break;
    case SPH_F16: ((__half*)out)[idx] = __float2half_rn(v); break;
    default: ((__nv_bfloat16*)out)[idx] = __float2bfloat16_rn(v);
  }
}

constexpr int kRows = 128;            // output rows of a tile
constexpr int kItem = 64;             // pairs of a step
constexpr int kBatch = 9;             // kernel offsets whose pair lists are held at a time

struct FfmaParams {
  const void* rows;
  const void* weight;                 // [KV, K, N]
  const int* nbr;                     // [KV, n_out]
  int64_t n_rows, n_out;
  int kv, K, N, flip_k, relu, out_dtype;
  int few, few_first;                 // conv_few_kernel's tiles: at most so many pairs, at most so many at the first kBatch
                                      // offsets; -1: it has none
  int walk_all;                       // conv_few_kernel takes every tile
  int w_vec;                          // filter rows can be read 4 elements at a time
  const float* scale;
  Bias bias;
  void* out;
  int* status;
};

// KC: input channels of a step, 32 (layers of at most 8 or 16 input channels: 8 or 16).
template <int CG, int KC> struct FfmaShape {
  static constexpr int NP = CG * 8;                  // output channels of a CTA, padded
  static constexpr int T = CG == 8 ? 128 : 64;       // threads of a CTA
  static constexpr int RL = T / CG;                  // row lanes
  static constexpr int RP = kItem / RL;              // rows per thread at most
  static constexpr int ACC = kRows * (NP + 4);       // floats
  static constexpr int AS = KC + 4;                  // floats of a staged row: 16-byte reads of 8 rows do not conflict
  static constexpr int A = kItem * AS;
  static constexpr int W = KC * NP;
  static constexpr int BYTES = (ACC + 2 * A + 2 * W) * 4 + kBatch * kRows * 5 + kBatch * 4;
  static constexpr bool PACKED = CG != 4;            // fma2
};

// Two fused multiply-adds, in one instruction (PACKED) or two; each is rounded as fmaf rounds.
template <bool PACKED = true>
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
  if (!PACKED) return make_float2(fmaf(a.x, b.x, c.x), fmaf(a.y, b.y, c.y));
  float2 d;
  asm("{\n\t.reg .b64 x, y, z;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\tmov.b64 z, {%6, %7};\n\t"
      "fma.rn.f32x2 z, x, y, z;\n\tmov.b64 {%0, %1}, z;\n\t}"
      : "=f"(d.x), "=f"(d.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
  return d;
}

// One step (offset, KC input channels) of RP rows x 8 output channels per thread.  The two 4-channel groups of a thread are
// NP/2 apart, so the lanes of a row read consecutive 16-byte pieces of the filter row.
template <int CG, int KC, int RP>
__device__ __forceinline__ void ffma_step(const float* __restrict__ a, const float* __restrict__ w, int kn, int rl, int cg,
                                          float2 (&acc)[FfmaShape<CG, KC>::RP][4]) {
  using S = FfmaShape<CG, KC>;
#pragma unroll 2
  for (int k4 = 0; k4 < kn; k4 += 4) {
    float av[RP][4];
#pragma unroll
    for (int j = 0; j < RP; ++j) {
      const float4 t = *(const float4*)(a + (rl + j * S::RL) * S::AS + k4);
      av[j][0] = t.x; av[j][1] = t.y; av[j][2] = t.z; av[j][3] = t.w;
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const float4 w0 = *(const float4*)(w + (k4 + q) * S::NP + cg * 4);
      const float4 w1 = *(const float4*)(w + (k4 + q) * S::NP + S::NP / 2 + cg * 4);
#pragma unroll
      for (int j = 0; j < RP; ++j) {
        const float2 x = make_float2(av[j][q], av[j][q]);
        acc[j][0] = fma2<S::PACKED>(x, make_float2(w0.x, w0.y), acc[j][0]);
        acc[j][1] = fma2<S::PACKED>(x, make_float2(w0.z, w0.w), acc[j][1]);
        acc[j][2] = fma2<S::PACKED>(x, make_float2(w1.x, w1.y), acc[j][2]);
        acc[j][3] = fma2<S::PACKED>(x, make_float2(w1.z, w1.w), acc[j][3]);
      }
    }
  }
}

// The calling thread's share of the tile's pairs at offsets k0 and up.  Out of line: few tiles get here, and inlined it costs
// the kernel registers and 3 % of its time.
__device__ __noinline__ int pairs_from(int k0, const int* __restrict__ nbr, int kv, int flip_k, int64_t n_out, int64_t n_rows,
                                       int64_t r0, int threads) {
  int n = 0;
  for (int k = k0; k < kv; ++k) {
    const int* col = nbr + (int64_t)(flip_k ? kv - 1 - k : k) * n_out + r0;
    for (int r = threadIdx.x; r < kRows; r += threads) {
      const int v = r0 + r < n_out ? __ldg(col + r) : -1;
      n += v >= 0 && v < n_rows;
    }
  }
  return n;
}

// A CTA owns 128 consecutive output rows x up to 64 output channels.  Per offset k the rows of the tile that have a
// neighbour are compacted into a list; up to 64 of their input rows and W[k] are staged (KC input channels a step, the next
// step's copies in flight), every thread multiplies ceil(pairs / row lanes) listed rows by 8 channels in registers, on top
// of the tile's fp32 accumulator in shared memory.  An output row occurs once per offset, so no two threads of a step hold the
// same accumulator.
// The CTA is small (64 or 128 threads) so that a thread has up to four rows: with one row per thread (256 threads a tile)
// the shared-memory reads of the filter, not the FMAs, set the pace; with eight rows too few warps fit on an SM.
// Bound by the shared-memory reads of the operands (74 % of that pipe).  Measured: 64 -> 64 on 170 k rows of 22 neighbours 3.2 ->
// 0.94 ms, 32 -> 32 on 390 k rows of 12 neighbours 1.9 -> 0.5 ms against the kernel it replaced (one thread group per row
// walking every slot of the table).  Two FMAs an instruction (fma2; the same bits) take the issue slots off its limits: 64 -> 64
// on 171 k rows 1070 -> 975 us, 32 -> 64 314 -> 292, 64 -> 16 on 472 k dense rows 1290 -> 1217; the weight gradient 845 -> 763, 228 -> 212,
// 511 -> 499.  Not in tiles of 32 output channels, which they make slower: 32 -> 32 on 5.4 k / 228 k rows 60 -> 65 / 265 -> 273 us,
// 16 -> 32 43 -> 47 / 165 -> 168, 128 -> 24 159 -> 173 / 733 -> 755.
// VEC: float32 rows of a multiple of 4 channels in and out, staged by 16-byte cp.async; else element by
// element.
template <typename T, int CG, int KC, bool VEC>
__global__ void __launch_bounds__(FfmaShape<CG, KC>::T) conv_ffma_kernel(FfmaParams p) {
  after_previous<false>();
  using S = FfmaShape<CG, KC>;
  extern __shared__ __align__(16) unsigned char smem[];
  float* s_acc = (float*)smem;                       // [kRows][NP + 4]
  float* s_a = s_acc + S::ACC;                       // [2][kItem][S::AS]
  float* s_w = s_a + 2 * S::A;                       // [2][KC][NP]
  int* s_in = (int*)(s_w + 2 * S::W);                // [kBatch][kRows] input row
  int* s_m = s_in + kBatch * kRows;                  // [kBatch] pairs
  unsigned char* s_out = (unsigned char*)(s_m + kBatch);   // [kBatch][kRows] row in the tile
  __shared__ int s_rest[S::T / 32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t r0 = (int64_t)blockIdx.x * kRows;
  const int n0 = blockIdx.y * S::NP;                 // first output channel of this CTA
  const int nc = min(S::NP, p.N - n0);
  const int rl = tid / CG, cg = tid % CG;
  const T* rows = (const T*)p.rows;
  const T* weight = (const T*)p.weight;
  const int k_chunks = (p.K + KC - 1) / KC;

  for (int e = tid; e < S::ACC; e += S::T) s_acc[e] = 0.f;

  auto stage = [&](int buf, int kb, int kk, int p0, int kc) {
    const int m = min(kItem, s_m[kk] - p0);
    const int* in = s_in + kk * kRows + p0;
    float* a = s_a + buf * S::A;
    float* w = s_w + buf * S::W;
    const T* wk = weight + ((int64_t)(kb + kk) * p.K + kc * KC) * p.N + n0;
    const int kn = min(KC, p.K - kc * KC);
    if constexpr (VEC) {
      const int c = tid % (KC / 4) * 4;
      const bool ok = c < kn;
      for (int r = tid / (KC / 4); r < m; r += S::T / (KC / 4)) {
        cp_async_16(smem_u32(a + r * S::AS + c), ok ? rows + (int64_t)in[r] * p.K + kc * KC + c : rows, ok ? 16u : 0u);
      }
      const int wc = tid % (S::NP / 4) * 4;
      const T* src = wk + (int64_t)(tid / (S::NP / 4)) * p.N + wc;
#pragma unroll 4
      for (int r = tid / (S::NP / 4); r < KC; r += S::T / (S::NP / 4)) {
        const bool ok = r < kn && wc < nc;
        cp_async_16(smem_u32(w + r * S::NP + wc), ok ? src : weight, ok ? 16u : 0u);
        src += (S::T / (S::NP / 4)) * p.N;
      }
    } else {
      for (int e = tid; e < m * KC; e += S::T) {
        const int r = e / KC, c = e % KC;
        stage_one(a + r * S::AS + c, c < kn ? rows + (int64_t)in[r] * p.K + kc * KC + c : rows, c < kn);
      }
      if (sizeof(T) == 4 && p.w_vec) {
        for (int e = tid; e < KC * S::NP / 4; e += S::T) {
          const int r = e / (S::NP / 4), c = e % (S::NP / 4) * 4;
          const bool ok = r < kn && c < nc;
          cp_async_16(smem_u32(w + r * S::NP + c), ok ? wk + (int64_t)r * p.N + c : weight, ok ? 16u : 0u);
        }
        return;
      }
      for (int e = tid; e < KC * S::NP; e += S::T) {
        const int r = e / S::NP, c = e % S::NP;
        const bool ok = r < kn && c < nc;
        stage_one(w + e, ok ? wk + (int64_t)r * p.N + c : weight, ok);
      }
    }
  };

  for (int kb = 0; kb < p.kv; kb += kBatch) {
    const int nk = min(kBatch, p.kv - kb);
    __syncthreads();                                  // the previous batch's lists are done with
    // kCols columns of the table at a time, all their loads in flight
    constexpr int kCols = 3;
    for (int k0 = warp; k0 < nk; k0 += kCols * (S::T / 32)) {
      int v[kCols][kRows / 32];
#pragma unroll
      for (int c = 0; c < kCols; ++c) {
        const int kk = k0 + c * (S::T / 32);
        const int* col = p.nbr + (int64_t)(p.flip_k ? p.kv - 1 - (kb + kk) : kb + kk) * p.n_out + r0;
#pragma unroll
        for (int h = 0; h < kRows / 32; ++h)
          v[c][h] = kk < nk && r0 + h * 32 + lane < p.n_out ? __ldg(col + h * 32 + lane) : -1;
      }
#pragma unroll
      for (int c = 0; c < kCols; ++c) {
        const int kk = k0 + c * (S::T / 32);
        if (kk >= nk) break;
        int n = 0;
#pragma unroll
        for (int h = 0; h < kRows / 32; ++h) {
          if (v[c][h] >= p.n_rows) {
            if (p.status) atomicOr(p.status, SPH_STATUS_BAD_INDEX);
            v[c][h] = -1;
          }
          const unsigned m = __ballot_sync(0xffffffffu, v[c][h] >= 0);
          if (v[c][h] >= 0) {
            const int pos = n + __popc(m & ((1u << lane) - 1u));
            s_in[kk * kRows + pos] = v[c][h];
            s_out[kk * kRows + pos] = (unsigned char)(h * 32 + lane);
          }
          n += __popc(m);
        }
        if (lane == 0) s_m[kk] = n;
      }
    }
    __syncthreads();
    if (kb == 0 && p.few >= 0) {                      // conv_few_kernel's tile?  By the same two counts, the same for all threads
      int n = 0;
      for (int k = 0; k < nk; ++k) n += s_m[k];
      if (n <= p.few_first) {
        n = pairs_from(nk, p.nbr, p.kv, p.flip_k, p.n_out, p.n_rows, r0, S::T);
        n = __reduce_add_sync(0xffffffffu, n);
        if (lane == 0) s_rest[warp] = n;
        __syncthreads();
        n = 0;
        for (int k = 0; k < nk; ++k) n += s_m[k];
        for (int w = 0; w < S::T / 32; ++w) n += s_rest[w];
        if (n <= p.few) return;
      }
    }
    int kk = 0, p0 = 0, kc = 0;
    while (kk < nk && s_m[kk] == 0) ++kk;
    if (kk < nk) stage(0, kb, kk, 0, 0);
    cp_async_commit();
    float2 acc[S::RP][4];
    for (int buf = 0; kk < nk; buf ^= 1) {
      int nkk = kk, np0 = p0, nkc = kc + 1;
      if (nkc == k_chunks) {
        nkc = 0;
        np0 += kItem;
        if (np0 >= s_m[kk]) {
          np0 = 0;
          do { ++nkk; } while (nkk < nk && s_m[nkk] == 0);
        }
      }
      cp_async_wait_pending(0);
      __syncthreads();       // the step's operands are there, everybody has left the other buffer and the accumulator
      if (nkk < nk) stage(buf ^ 1, kb, nkk, np0, nkc);
      cp_async_commit();
      const int m = min(kItem, s_m[kk] - p0);
      // the accumulator tile is read before an item and written behind it: an output is ONE chain of fused multiply-adds
      // over the offsets and input channels in ascending order, whatever the tiling
      auto tile_row = [&](int r) { return s_acc + (int)s_out[kk * kRows + p0 + r] * (S::NP + 4) + cg * 4; };
      if (kc == 0) {
#pragma unroll
        for (int j = 0; j < S::RP; ++j) {
          if (rl + j * S::RL < m) {
            const float* d = tile_row(rl + j * S::RL);
            const float4 t0 = *(const float4*)d, t1 = *(const float4*)(d + S::NP / 2);
            acc[j][0] = make_float2(t0.x, t0.y); acc[j][1] = make_float2(t0.z, t0.w);
            acc[j][2] = make_float2(t1.x, t1.y); acc[j][3] = make_float2(t1.z, t1.w);
          }
        }
      }
      const float* a = s_a + buf * S::A;
      const float* w = s_w + buf * S::W;
      // rows beyond m are staged rows of an earlier step: multiplied, never added
      const int rp = (m + S::RL - 1) / S::RL;
      // what is staged beyond K is zero; a bound the compiler knows costs full steps nothing (32 -> 64: 240 against 249 us)
      const int kn = VEC ? KC : (min(KC, p.K - kc * KC) + 7) & ~7;
      switch (rp) {
        case 1: ffma_step<CG, KC, 1>(a, w, kn, rl, cg, acc); break;
        case 2: ffma_step<CG, KC, (S::RP < 2 ? 1 : 2)>(a, w, kn, rl, cg, acc); break;
        case 3: ffma_step<CG, KC, (S::RP < 3 ? 1 : 3)>(a, w, kn, rl, cg, acc); break;
        default: ffma_step<CG, KC, (S::RP < 4 ? 1 : 4)>(a, w, kn, rl, cg, acc);
      }
      if (kc == k_chunks - 1) {
#pragma unroll
        for (int j = 0; j < S::RP; ++j) {
          if (rl + j * S::RL < m) {
            float* d = tile_row(rl + j * S::RL);
            *(float4*)d = make_float4(acc[j][0].x, acc[j][0].y, acc[j][1].x, acc[j][1].y);
            *(float4*)(d + S::NP / 2) = make_float4(acc[j][2].x, acc[j][2].y, acc[j][3].x, acc[j][3].y);
          }
        }
      }
      kk = nkk; p0 = np0; kc = nkc;
    }
  }
  __syncthreads();
  const int rows_here = (int)min((int64_t)kRows, p.n_out - r0);
  for (int e = tid; e < rows_here * nc; e += S::T) {
    const int r = e / nc, c = e % nc;
    float v = s_acc[r * (S::NP + 4) + c];
    if (p.scale) v *= __ldg(p.scale + n0 + c);
    if (p.bias.data) v += p.bias.at<sizeof(T) == 2>(n0 + c);
    store_one(p.out, p.out_dtype, (r0 + r) * p.N + n0 + c, p.relu ? fmaxf(v, 0.f) : v);
  }
}

// ---- tiles with few pairs ------------------------------------------------------------------------------------------
// A staged step costs its filter slice and a barrier whether it serves 2 pairs or 64, and the tile's buffers leave room for
// a few hundred threads on an SM.  Below some pairs a row it is faster to have every row walked by threads of its own (4
// output channels each), straight from global memory: nothing is shared, so the machine is full of independent chains of
// loads, which is all that bounds them.  The two launches share the tiles: each counts a tile's pairs and takes it or leaves it.
// Rules and forward of a layer on 78 k rows of 1.5 neighbours, row walks for all tiles -> staged only -> both: 64 -> 64
// 200 -> 220 -> 155 us, with stride 2 717 -> 537 -> 390; 37 -> 64 fp16 with stride 2 514 -> 623 -> 260.  A training step of the
// fp32 encoder, whose deeper levels are dense, takes 11.8 ms either way.
// Layers of which no tile is better staged (launch_ffma_cg says which) are walked in one launch that counts nothing.
// The tile's table entries are read once, into shared memory, with a bit per present offset.
constexpr int kFewThreads = 512;
constexpr int kFewSmem = 200 * 1024;  // entries and bits of a tile: up to 387 offsets

// 16-bit values by the builtin load of an integer: the one of a __half is an asm statement, which the compiler may move in
// front of the check that guards it.
__device__ __forceinline__ float load_f(const float* p) { return __ldg(p); }
__device__ __forceinline__ float load_f(const __half* p) { return __half2float(__ushort_as_half(__ldg((const unsigned short*)p))); }
__device__ __forceinline__ float load_f(const __nv_bfloat16* p) {
  return __uint_as_float((uint32_t)__ldg((const unsigned short*)p) << 16);
}

__device__ __forceinline__ void load_f4(const float* p, float (&v)[4]) {
  const float4 t = __ldg((const float4*)p);
  v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
}
__device__ __forceinline__ void load_f4(const __half* p, float (&v)[4]) {
  const uint2 t = __ldg((const uint2*)p);
  const float2 a = __half22float2(*(const __half2*)&t.x), b = __half22float2(*(const __half2*)&t.y);
  v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
}
__device__ __forceinline__ void load_f4(const __nv_bfloat16* p, float (&v)[4]) {
  const uint2 t = __ldg((const uint2*)p);
  const float2 a = __bfloat1622float2(*(const __nv_bfloat162*)&t.x), b = __bfloat1622float2(*(const __nv_bfloat162*)&t.y);
  v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
}

// acc[0..3] += x[0..K) W[:, 0..3], input channels ascending (the order of ffma_step).  XV / WV: four elements of the input /
// filter row a load.
template <typename T, bool XV, bool WV>
__device__ __forceinline__ void add_pair(const T* __restrict__ x, const T* __restrict__ w, int K, int N, float (&acc)[4]) {
  int k = 0;
#pragma unroll 2
  for (; k + 4 <= K; k += 4) {
    float xv[4], wv[4][4];
    if constexpr (XV) load_f4(x + k, xv);
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      if constexpr (!XV) xv[u] = load_f(x + k + u);
      if constexpr (WV) {
        load_f4(w + (k + u) * N, wv[u]);
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j) wv[u][j] = load_f(w + (k + u) * N + j);
      }
    }
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[j] = fmaf(xv[u], wv[u][j], acc[j]);
  }
#pragma unroll 1
  for (; k < K; ++k) {
    const float xv = load_f(x + k);
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[j] = fmaf(xv, load_f(w + k * N + j), acc[j]);
  }
}

template <typename T, bool XV, bool WV>
__global__ void __launch_bounds__(kFewThreads, 2) conv_few_kernel(FfmaParams p) {
  after_previous<false>();
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ int s_count[kFewThreads / 32];
  const int words = (p.kv + 31) / 32;
  int* s_entry = (int*)smem;                         // [kv][kRows]
  unsigned* s_present = (unsigned*)(s_entry + p.kv * kRows);   // [words][kRows], bit k: the row has a neighbour at offset k
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t r0 = (int64_t)blockIdx.x * kRows;
  const int r = tid % kRows;
  for (int e = tid; e < words * kRows; e += kFewThreads) s_present[e] = 0u;
  __syncthreads();
  int n = 0;
  auto entry = [&](int k) {
    const int v = r0 + r < p.n_out ? __ldg(p.nbr + (int64_t)(p.flip_k ? p.kv - 1 - k : k) * p.n_out + r0 + r) : -1;
    if (v >= p.n_rows) {
      if (p.status) atomicOr(p.status, SPH_STATUS_BAD_INDEX);
    } else if (v >= 0) {
      s_entry[k * kRows + r] = v;
      atomicOr(s_present + k / 32 * kRows + r, 1u << (k & 31));
      ++n;
    }
  };
  auto pairs = [&]() {                               // the CTA's, so far
    const int mine = __reduce_add_sync(0xffffffffu, n);
    __syncthreads();                                 // the last sum has been read
    if (lane == 0) s_count[warp] = mine;
    __syncthreads();
    int sum = 0;
#pragma unroll
    for (int w = 0; w < kFewThreads / 32; ++w) sum += s_count[w];
    return sum;
  };
  constexpr int STEP = kFewThreads / kRows;
  const int first = p.walk_all ? 0 : min(kBatch, p.kv);
  if (!p.walk_all) {
#pragma unroll
    for (int h = 0; h < (kBatch + STEP - 1) / STEP; ++h)
      if (tid / kRows + h * STEP < first) entry(tid / kRows + h * STEP);
    if (pairs() > p.few_first) return;
  }
#pragma unroll 7
  for (int k = first + tid / kRows; k < p.kv; k += STEP) entry(k);
  if (p.walk_all) __syncthreads();
  else if (pairs() > p.few) return;
  const int groups = (p.N + 3) / 4;
  const int rows_here = (int)min((int64_t)kRows, p.n_out - r0);
  const T* weight = (const T*)p.weight;
  for (int e = tid; e < rows_here * groups; e += kFewThreads) {
    const int row = e / groups, c = min(e % groups * 4, p.N - 4);   // the last two of an odd width share columns: the same values
    float acc[4] = {0.f, 0.f, 0.f, 0.f};
    for (int w = 0; w < words; ++w) {
      for (unsigned m = s_present[w * kRows + row]; m; m &= m - 1) {
        const int k = w * 32 + __ffs(m) - 1;
        const int i = s_entry[k * kRows + row];
        add_pair<T, XV, WV>((const T*)p.rows + (int64_t)i * p.K, weight + (int64_t)k * p.K * p.N + c, p.K, p.N, acc);
      }
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      float v = acc[j];
      if (p.scale) v *= __ldg(p.scale + c + j);
      if (p.bias.data) v += p.bias.at<sizeof(T) == 2>(c + j);
      store_one(p.out, p.out_dtype, (r0 + row) * p.N + c + j, p.relu ? fmaxf(v, 0.f) : v);
    }
  }
}

// ---- weight gradient: dW[k] += X_i^T dY_o over the pairs of offset k ------------------------------------------------
// grid (row slices, KV).  A CTA compacts the pairs of its slice, then stages PAIRS of them at a time (the next ones'
// copies in flight); a thread owns 8 input x 8 output channels of the product, the threads are as many copies of the
// K x N tile as fit, and each copy takes its share of the staged pairs.  The copies are summed in shared memory and added
// to the gradient once per CTA.
constexpr int kThreads = 256;
constexpr int kWgSlice = 2048;
constexpr int kWgMaxCh = 64;

struct FfmaWgradParams {
  const void* rows;                   // [n_rows, K]
  const void* dout;                   // [n_out, N]
  const int* nbr;                     // [KV, n_out]
  int64_t n_rows, n_out;
  int K, N;
  float* dw;                          // [KV, K, N], accumulated into
  int* status;
};

// KG / NG: groups of 8 channels on either side.
template <int KG, int NG> struct WgShape {
  static constexpr int XS = KG * 8 + 4, DS = NG * 8 + 4;     // staged row strides in floats
  static constexpr int COPIES = kThreads / (KG * NG);
  static constexpr int PAIRS = COPIES > 32 ? COPIES : 32;    // staged at a time: one for every copy at least
  static constexpr int STAGE = PAIRS * (XS + DS);            // floats
  static constexpr int RED = KG * NG * 64;                   // floats of the product
  static constexpr int BYTES = (2 * STAGE > RED ? 2 * STAGE : RED) * 4 + kWgSlice * 8 + 64;
};

// Sums LEFT products a lane over the lanes that differ in the bits O, 2 O .. 16, each exchange halving what a lane holds (it
// keeps the half its bit names).  Returns the first product that v[0] now stands for.  A serial pass over 256 copies of a
// 5 x 5 layer took longer than its products (78 k rows of 1.5 neighbours: 377 -> 19 us; 64 -> 7: 165 -> 74 us).
template <int O, int LEFT>
__device__ __forceinline__ int fold_copies(float (&v)[64], int lane) {
  if constexpr (O < 32) {
    const bool up = (lane & O) != 0;
#pragma unroll
    for (int j = 0; j < LEFT / 2; ++j) {
      const float got = __shfl_xor_sync(0xffffffffu, up ? v[j] : v[j + LEFT / 2], O);
      v[j] = (up ? v[j + LEFT / 2] : v[j]) + got;
    }
    return (up ? LEFT / 2 : 0) + fold_copies<O * 2, LEFT / 2>(v, lane);
  } else {
    return 0;
  }
}

template <typename T, int KG, int NG, bool VEC>
__global__ void __launch_bounds__(kThreads, 2) conv_wgrad_ffma_kernel(FfmaWgradParams p) {
  after_previous<false>();
  using S = WgShape<KG, NG>;
  extern __shared__ __align__(16) unsigned char smem[];
  float* s_st = (float*)smem;                                // [2]{x [PAIRS][XS], dy [PAIRS][DS]}, later the sum
  int* s_in = (int*)(smem + (2 * S::STAGE > S::RED ? 2 * S::STAGE : S::RED) * 4);
  int* s_out = s_in + kWgSlice;
  int* s_cnt = s_out + kWgSlice;                             // [8] hits per warp
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int k = blockIdx.y;
  const int64_t r0 = (int64_t)blockIdx.x * kWgSlice;
  const int nr = (int)min((int64_t)kWgSlice, p.n_out - r0);
  const T* rows = (const T*)p.rows;
  const T* dout = (const T*)p.dout + r0 * p.N;

  // compaction in ascending row order: a warp's eighth of the slice stays in registers between the count and the write
  constexpr int kPer = kWgSlice / kThreads;                  // 32-row chunks per warp
  const int* col = p.nbr + (int64_t)k * p.n_out + r0 + warp * (kPer * 32);
  int v[kPer], cnt = 0;
#pragma unroll
  for (int h = 0; h < kPer; ++h) v[h] = warp * (kPer * 32) + h * 32 + lane < nr ? __ldg(col + h * 32 + lane) : -1;
#pragma unroll
  for (int h = 0; h < kPer; ++h) {
    if (v[h] >= p.n_rows) {
      if (p.status) atomicOr(p.status, SPH_STATUS_BAD_INDEX);
      v[h] = -1;
    }
    cnt += __popc(__ballot_sync(0xffffffffu, v[h] >= 0));
  }
  if (lane == 0) s_cnt[warp] = cnt;
  __syncthreads();
  int at = 0, n = 0;
  for (int w = 0; w < kThreads / 32; ++w) {
    if (w < warp) at += s_cnt[w];
    n += s_cnt[w];
  }
  if (n == 0) return;
#pragma unroll
  for (int h = 0; h < kPer; ++h) {
    const unsigned m = __ballot_sync(0xffffffffu, v[h] >= 0);
    if (v[h] >= 0) {
      const int pos = at + __popc(m & ((1u << lane) - 1u));
      s_in[pos] = v[h];
      s_out[pos] = warp * (kPer * 32) + h * 32 + lane;
    }
    at += __popc(m);
  }
  __syncthreads();

  auto stage = [&](int buf, int p0) {
    float* x = s_st + buf * S::STAGE;
    float* d = x + S::PAIRS * S::XS;
    const int np = min(S::PAIRS, n - p0);
    if constexpr (VEC) {
      for (int e = tid; e < S::PAIRS * KG * 2; e += kThreads) {
        const int r = e / (KG * 2), c = (e % (KG * 2)) * 4;
        const bool ok = r < np && c < p.K;
        cp_async_16(smem_u32(x + r * S::XS + c), ok ? rows + (int64_t)s_in[p0 + r] * p.K + c : rows, ok ? 16u : 0u);
      }
      for (int e = tid; e < S::PAIRS * NG * 2; e += kThreads) {
        const int r = e / (NG * 2), c = (e % (NG * 2)) * 4;
        const bool ok = r < np && c < p.N;
        cp_async_16(smem_u32(d + r * S::DS + c), ok ? dout + (int64_t)s_out[p0 + r] * p.N + c : dout, ok ? 16u : 0u);
      }
    } else {
      for (int e = tid; e < S::PAIRS * KG * 8; e += kThreads) {
        const int r = e / (KG * 8), c = e % (KG * 8);
        const bool ok = r < np && c < p.K;
        stage_one(x + r * S::XS + c, ok ? rows + (int64_t)s_in[p0 + r] * p.K + c : rows, ok);
      }
      for (int e = tid; e < S::PAIRS * NG * 8; e += kThreads) {
        const int r = e / (NG * 8), c = e % (NG * 8);
        const bool ok = r < np && c < p.N;
        stage_one(d + r * S::DS + c, ok ? dout + (int64_t)s_out[p0 + r] * p.N + c : dout, ok);
      }
    }
  };

  const int copy = tid / (KG * NG), in_copy = tid % (KG * NG);
  const int ig = in_copy / NG, og = in_copy % NG;
  float2 pairs[32];                                          // [8 input][4 x 2 output channels]
#pragma unroll
  for (int i = 0; i < 32; ++i) pairs[i] = make_float2(0.f, 0.f);
  stage(0, 0);
  cp_async_commit();
  int buf = 0;
  for (int p0 = 0; p0 < n; p0 += S::PAIRS, buf ^= 1) {
    cp_async_wait_pending(0);
    __syncthreads();
    if (p0 + S::PAIRS < n) stage(buf ^ 1, p0 + S::PAIRS);
    cp_async_commit();
    const float* x = s_st + buf * S::STAGE + ig * 8;
    const float* d = s_st + buf * S::STAGE + S::PAIRS * S::XS + og * 4;
    const int np = min(S::PAIRS, n - p0);
#pragma unroll 2
    for (int r = copy; r < np; r += S::COPIES) {
      const float4 x0 = *(const float4*)(x + r * S::XS), x1 = *(const float4*)(x + r * S::XS + 4);
      // the thread's output channels: 4 og .. 4 og + 3 of either half, so that the lanes read consecutive pieces
      const float4 d0 = *(const float4*)(d + r * S::DS), d1 = *(const float4*)(d + r * S::DS + NG * 4);
      const float xv[8] = {x0.x, x0.y, x0.z, x0.w, x1.x, x1.y, x1.z, x1.w};
      const float2 dv[4] = {make_float2(d0.x, d0.y), make_float2(d0.z, d0.w), make_float2(d1.x, d1.y), make_float2(d1.z, d1.w)};
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) pairs[i * 4 + j] = fma2(make_float2(xv[i], xv[i]), dv[j], pairs[i * 4 + j]);
    }
  }
  float acc[64];                                             // [8 input][8 output channels]
#pragma unroll
  for (int i = 0; i < 32; ++i) {
    acc[2 * i] = pairs[i].x;
    acc[2 * i + 1] = pairs[i].y;
  }
  // Sum of the copies: those of a warp in its registers, then the warps' (or the wider copies') one after the other.
  constexpr int kLanes = KG * NG < 32 ? KG * NG : 32;        // lanes of a warp that hold one copy
  constexpr int kLeft = 64 * kLanes / 32;                    // products a lane is left with: acc[0 .. kLeft) are first ..
  const int first = fold_copies<kLanes, 64>(acc, lane);
  float* red = s_st;
  constexpr int kSums = KG * NG < 32 ? kThreads / 32 : S::COPIES;
  const int mine = KG * NG < 32 ? warp : copy;
  for (int c = 0; c < kSums; ++c) {
    __syncthreads();
    if (mine == c) {
#pragma unroll
      for (int e = 0; e < kLeft; ++e) {
        const int i = (first + e) / 8, j = (first + e) % 8;
        float* t = red + (ig * 8 + i) * (NG * 8) + (j < 4 ? 0 : NG * 4) + og * 4 + (j & 3);
        *t = c == 0 ? acc[e] : *t + acc[e];
      }
    }
  }
  __syncthreads();
  float* dw = p.dw + (int64_t)k * p.K * p.N;
  for (int e = tid; e < p.K * p.N; e += kThreads) atomicAdd(dw + e, red[(e / p.N) * (NG * 8) + e % p.N]);
}

template <typename T, int CG, int KC, bool VEC>
int launch_ffma(const FfmaParams& p, cudaStream_t st) {
  using S = FfmaShape<CG, KC>;
  auto kern = conv_ffma_kernel<T, CG, KC, VEC>;
  SPH_CUDA(allow_smem(kern, S::BYTES));
  const dim3 grid((unsigned)div_up64(p.n_out, kRows), (unsigned)div_up(p.N, S::NP));
  launch(kern, grid, S::T, S::BYTES, st, p);
  SPH_LAUNCH_CHECK();
  return SPH_OK;
}

template <typename T, bool XV, bool WV>
int launch_few(const FfmaParams& p, int smem, cudaStream_t st) {
  auto kern = conv_few_kernel<T, XV, WV>;
  SPH_CUDA(allow_smem(kern, kFewSmem));
  launch(kern, (unsigned)div_up64(p.n_out, kRows), kFewThreads, smem, st, p);
  SPH_LAUNCH_CHECK();
  return SPH_OK;
}

template <typename T, int KC, bool VEC>
int launch_ffma_cg(FfmaParams p, cudaStream_t st) {
  p.w_vec = p.N % 4 == 0 && ((uintptr_t)p.weight & (4 * sizeof(T) - 1)) == 0;
  const bool x_vec = p.K % 4 == 0 && ((uintptr_t)p.rows & (4 * sizeof(T) - 1)) == 0;
  const int sms = current_sm_count();
  if (sms <= 0) return SPH_ERR_CUDA;
  const int smem = (p.kv + (p.kv + 31) / 32) * kRows * 4;
  // What a staged tile multiplies beyond its channels: K in steps of KC, N in tiles of 8, 16, 32 or 64.
  const int np = p.N <= 8 ? 8 : p.N <= 16 ? 16 : p.N <= 32 ? 32 : div_up(p.N, 64) * 64;
  const double waste = (double)(div_up(p.K, KC) * KC) / p.K * np / p.N;
  const bool small = div_up64(p.n_out, kRows) <= 4 * (int64_t)sms;     // few CTAs to hide a CTA's steps behind
  // All tiles are walked where padding makes every staged step dear: 16-bit rows (a conversion each; 48 -> 40 at 1.3 to 15 neighbours a
  // row 872 -> 313 to 4207 -> 3239 us; not with filter rows read by the element: 64 -> 33 at 9.4 3063 -> 5883), float32 rows of 9 to 16 channels staged element by element (9 -> 16: 139 -> 87, 565 -> 432),
  // small float32 layers (3 -> 16 on 23 k rows 48 -> 19, 24 -> 40 on 67 k rows 183 -> 122; on 531 k rows 939 -> 1119).
  const bool can = p.N >= 4 && smem <= kFewSmem;
  const bool padded = waste >= 1.5;
  p.walk_all = can && padded && ((p.w_vec && (sizeof(T) == 2 || (!VEC && p.K > 8 && p.K <= 16))) ||
                                 (sizeof(T) == 4 && small && (p.kv > kBatch || p.K > 8)));
  // Else two pairs a row for 27 offsets (in large layers as many for an offset of larger filters: 32 -> 32 at 45 offsets and 2.5
  // pairs a row 548 -> 452 us), by a count of all offsets for the tiles that have few at the first ones.  (By the first ones alone
  // the top row of a scan, which has no neighbours above it, would pass; by all of them alone every dense tile would pay for the
  // count.)  A limit of three costs a 64 -> 64 training layer on 103 k rows 774 -> 984 us of convolution kernels.  Large layers of
  // 16-bit rows, staged at a conversion an element: four (64 -> 64 at 45 offsets and 2.5 pairs a row 1424 -> 802 us).  Rows of
  // up to 16 channels and products of up to 8 are staged in any case: their steps are short.
  p.few = p.few_first = -1;
  if (can && !p.walk_all && p.K > 16 && p.N > 8) {
    const double more = p.kv > 27 && !small && sizeof(T) == 4 ? p.kv / 27.0 : 1.0;
    const bool dear = sizeof(T) == 2 && !small && p.w_vec;
    p.few = (int)(kRows * (dear ? 4 : VEC ? 2 : 2.5) * more);
    p.few_first = p.kv <= kBatch ? p.few : dear ? kRows * 3 / 2 : kRows * 3 / 4;
  }
  if (p.walk_all || p.few >= 0) {
    int rc;
    if (x_vec && p.w_vec) rc = launch_few<T, true, true>(p, smem, st);
    else if (p.w_vec) rc = launch_few<T, false, true>(p, smem, st);
    else rc = launch_few<T, false, false>(p, smem, st);
    if (rc != SPH_OK || p.walk_all) return rc;
  }
  // the narrowest tile that holds the output channels; beyond 64 of them the grid repeats the rows per 64
  if (p.N <= 8) return launch_ffma<T, 1, KC, VEC>(p, st);
  if (p.N <= 16) return launch_ffma<T, 2, KC, VEC>(p, st);
  if (p.N <= 32) return launch_ffma<T, 4, KC, VEC>(p, st);
  return launch_ffma<T, 8, KC, VEC>(p, st);
}

// Narrow float32 rows take a step as wide as they are: the zeros that would fill it to 32 channels cost as many issue slots
// as channels do, and the smaller buffers let more CTAs reside (sparse layers are bound by the latency of their
// steps).  Four buffers instead of two are slower (16 -> 32, 78 k rows: 46 -> 72 us).
template <bool VEC>
int launch_ffma_f32(const FfmaParams& p, cudaStream_t st) {
  if (p.K <= 8) return launch_ffma_cg<float, 8, VEC>(p, st);
  if (p.K <= 16) return launch_ffma_cg<float, 16, VEC>(p, st);
  return launch_ffma_cg<float, 32, VEC>(p, st);
}

template <typename T, int KG, int NG, bool VEC>
int launch_wg(const FfmaWgradParams& p, int kv, cudaStream_t st) {
  using S = WgShape<KG, NG>;
  auto kern = conv_wgrad_ffma_kernel<T, KG, NG, VEC>;
  SPH_CUDA(allow_smem(kern, S::BYTES));
  launch(kern, dim3((unsigned)div_up64(p.n_out, kWgSlice), (unsigned)kv), kThreads, S::BYTES, st, p);
  SPH_LAUNCH_CHECK();
  return SPH_OK;
}

template <typename T, int KG, bool VEC>
int launch_wg_n(const FfmaWgradParams& p, int kv, cudaStream_t st) {
  if (p.N <= 8) return launch_wg<T, KG, 1, VEC>(p, kv, st);
  if (p.N <= 16) return launch_wg<T, KG, 2, VEC>(p, kv, st);
  if (p.N <= 32) return launch_wg<T, KG, 4, VEC>(p, kv, st);
  return launch_wg<T, KG, 8, VEC>(p, kv, st);
}

template <typename T, bool VEC>
int launch_wg_k(const FfmaWgradParams& p, int kv, cudaStream_t st) {
  if (p.K <= 8) return launch_wg_n<T, 1, VEC>(p, kv, st);
  if (p.K <= 16) return launch_wg_n<T, 2, VEC>(p, kv, st);
  if (p.K <= 32) return launch_wg_n<T, 4, VEC>(p, kv, st);
  return launch_wg_n<T, 8, VEC>(p, kv, st);
}

}  // namespace

int conv_gather_ffma(const void* rows, int dtype, int64_t n_rows, const void* weight, const int* nbr, int64_t n_out,
                     int kv, int K, int N, int flip_k, const float* scale, Bias bias, int relu, void* out,
                     int out_dtype, int* status, cudaStream_t st) {
  FfmaParams p;
  p.rows = rows; p.weight = weight; p.nbr = nbr;
  p.n_rows = n_rows; p.n_out = n_out;
  p.kv = kv; p.K = K; p.N = N; p.flip_k = flip_k; p.relu = relu; p.out_dtype = out_dtype;
  p.scale = scale; p.bias = bias; p.out = out; p.status = status;
  switch (dtype) {
    case SPH_F32:
      if (K % 4 == 0 && N % 4 == 0 && (((uintptr_t)rows | (uintptr_t)weight) & 15u) == 0)
        return launch_ffma_f32<true>(p, st);
      return launch_ffma_f32<false>(p, st);
    case SPH_F16: return launch_ffma_cg<__half, 32, false>(p, st);
    case SPH_BF16: return launch_ffma_cg<__nv_bfloat16, 32, false>(p, st);
  }
  set_error("unknown dtype %d", dtype);
  return SPH_ERR_INVALID;
}

int conv_wgrad_ffma(const void* rows, const void* dout, int dtype, int64_t n_rows, const int* nbr, int64_t n_out, int kv,
                    int K, int N, float* dw, int* status, cudaStream_t st) {
  if (K > kWgMaxCh || N > kWgMaxCh) {
    set_error("weight gradient supports up to %d channels (got %d x %d)", kWgMaxCh, K, N);
    return SPH_ERR_LIMIT;
  }
  FfmaWgradParams p;
  p.rows = rows; p.dout = dout; p.nbr = nbr;
  p.n_rows = n_rows; p.n_out = n_out;
  p.K = K; p.N = N; p.dw = dw; p.status = status;
  switch (dtype) {
    case SPH_F32:
      if (K % 4 == 0 && N % 4 == 0 && (((uintptr_t)rows | (uintptr_t)dout) & 15u) == 0)
        return launch_wg_k<float, true>(p, kv, st);
      return launch_wg_k<float, false>(p, kv, st);
    case SPH_F16: return launch_wg_k<__half, false>(p, kv, st);
    case SPH_BF16: return launch_wg_k<__nv_bfloat16, false>(p, kv, st);
  }
  set_error("weight gradient is not defined for dtype %d", dtype);
  return SPH_ERR_UNSUPPORTED;
}

}  // namespace sph
