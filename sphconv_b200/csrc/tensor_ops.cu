// COO <-> range-voxel <-> dense: the tensor operations on either side of the convolution path.
//
// The reference (src/sphconv/tensor.cu) builds a dense int32 grid [B,H,W,D] to count the voxels of every column
// (fillGridKernel + torch::sum + cumsum, tensor.cu:96-109), places the rows with one atomic per voxel (order inside a
// column = arrival order, tensor.cu:55-76) and hard-codes float.  Here the grid is one BIT per voxel (a depth bitmask
// per column), a voxel's row is "column start + set bits below its depth" - no atomics on positions, rows of a column
// come out in ascending depth (what the rule kernels' column index wants) - and rows are copied as bytes, so every
// dtype goes through the same kernels.
#include "common.cuh"

namespace sph {

namespace {

constexpr int kOpsThreads = 256;

__device__ __forceinline__ int col_begin(const int* __restrict__ zp, int64_t c) { return c == 0 ? 0 : __ldg(zp + c - 1); }

// indices [nnz][4] = (b, s0, s1, s2).  Sets the voxel's bit; out-of-range coordinates raise the status bit.
__global__ void __launch_bounds__(kOpsThreads)
mark_voxels_kernel(const int* __restrict__ idx, int64_t nnz, int B, int H, int W, int D, int words,
                   uint32_t* __restrict__ mask, int* __restrict__ status) {
  after_previous();
  const int64_t n = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= nnz) return;
  const int4 v = __ldg((const int4*)idx + n);
  if ((unsigned)v.x >= (unsigned)B || (unsigned)v.y >= (unsigned)H || (unsigned)v.z >= (unsigned)W ||
      (unsigned)v.w >= (unsigned)D) {
    if (status) atomicOr(status, SPH_STATUS_BAD_INDEX);
    return;
  }
  const int64_t col = ((int64_t)v.x * H + v.y) * W + v.z;
  atomicOr(mask + col * words + (v.w >> 5), 1u << (v.w & 31));
}

// Row of every COO entry: column start + number of set bits below its depth.
__global__ void __launch_bounds__(kOpsThreads)
place_voxels_kernel(const int* __restrict__ idx, int64_t nnz, int B, int H, int W, int D, int words,
                    const uint32_t* __restrict__ mask, const int* __restrict__ z_ptr, int* __restrict__ z_idx,
                    int* __restrict__ permutation) {
  after_previous();
  const int64_t n = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= nnz) return;
  const int4 v = __ldg((const int4*)idx + n);
  if ((unsigned)v.x >= (unsigned)B || (unsigned)v.y >= (unsigned)H || (unsigned)v.z >= (unsigned)W ||
      (unsigned)v.w >= (unsigned)D) {
    permutation[n] = -1;
    return;
  }
  const int64_t col = ((int64_t)v.x * H + v.y) * W + v.z;
  const uint32_t* m = mask + col * words;
  int below = 0;
  const int w_hit = v.w >> 5;
  for (int w = 0; w < w_hit; ++w) below += __popc(__ldg(m + w));
  below += __popc(__ldg(m + w_hit) & ((1u << (v.w & 31)) - 1u));
  const int pos = col_begin(z_ptr, col) + below;
  permutation[n] = pos;
  z_idx[pos] = v.w;
}

// dst[perm[n]] = src[n] (scatter) or dst[n] = src[perm[n]] (gather); rows of `row_bytes` bytes copied in pieces of
// `piece` bytes (16, 4, 2 or 1, whatever divides the row and the base addresses).
template <typename V>
__global__ void __launch_bounds__(kOpsThreads)
permute_rows_kernel(const V* __restrict__ src, V* __restrict__ dst, const int* __restrict__ perm, int64_t n_rows,
                    int pieces, int gather) {
  after_previous();
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t n = t / pieces;
  const int c = (int)(t % pieces);
  if (n >= n_rows) return;
  const int p = __ldg(perm + n);
  if (p < 0) return;
  if (gather) dst[n * pieces + c] = src[(int64_t)p * pieces + c];
  else dst[(int64_t)p * pieces + c] = src[n * pieces + c];
}

// Range-voxel rows <-> dense [B,H,W,D,C]: the row's column is found by a search in z_ptr.
template <typename V>
__global__ void __launch_bounds__(kOpsThreads)
dense_rows_kernel(V* __restrict__ rows, const int* __restrict__ z_idx, const int* __restrict__ z_ptr, int64_t nnz,
                  int64_t ncols, int D, int pieces, V* __restrict__ dense, int backward, int* __restrict__ status) {
  after_previous();
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t n = t / pieces;
  const int c = (int)(t % pieces);
  if (n >= nnz) return;
  int64_t lo = 0, hi = ncols - 1;          // first column whose inclusive prefix exceeds n
  while (lo < hi) {
    const int64_t mid = (lo + hi) >> 1;
    if (__ldg(z_ptr + mid) > n) hi = mid; else lo = mid + 1;
  }
  const int z = __ldg(z_idx + n);
  if ((unsigned)z >= (unsigned)D) {
    if (status) atomicOr(status, SPH_STATUS_BAD_INDEX);
    return;
  }
  const int64_t off = ((lo * D + z) * pieces) + c;
  if (backward) rows[n * pieces + c] = dense[off];
  else dense[off] = rows[n * pieces + c];
}

// Rows <-> dense [B,C,H,W,D], channels first: what a convolution head reads.  A block takes whole columns (consecutive
// columns are consecutive rows AND consecutive dense cells of every channel), stages their rows in shared memory with a
// cell -> row map, and moves every channel's cells in vectors of V elements; cells without a row are zeros.  The dense
// tensor is written once; a fill, a channels-last scatter and a permuting copy moved its bytes four times.  [8,64,16,128,64]
// fp16 (134 MB) with 30 % of the cells occupied: 58 us to dense and 53 us back against 350 and 325 us; DRAM is 22 and 40 % busy,
// the rest is the per-element traffic of the staged rows.
//
// Rows need not own their cells: of several rows at one depth of a column the last is the cell's value and each gets the
// cell's gradient; a row whose depth lies outside the grid has the status bit set and a gradient of zero.  A block can hence have
// more rows than cells (`crowded`): shared memory then holds one row per cell, the one its value comes from.
constexpr int kDenseCells = 256;         // cells of a block, when columns are shorter and rows not narrow
constexpr int kDenseMaxCells = 2048;     // columns up to this deep are staged
// Narrow rows on large grids: more cells a block, up to this many bytes if all are occupied and while this many blocks are left.  Blocks
// of 256 cells with a few words for each are bound by the two round trips to memory of every block: 33.5 M cells, 284 k rows, one
// float32 channel 324 -> 56 us and 333 -> 61 back, 12 int8 channels 686 -> 293 and 659 -> 249.
constexpr int64_t kDenseBytes = 16384;
constexpr int64_t kDenseBlocks = 16 * 148;
constexpr int kDenseSmem = 96 * 1024;    // the cells' map (8 KB), 64 KB of rows, and at most 8 bytes a row of padding

// Rows of `words` pieces between memory (pitch words apart) and shared memory (s_pitch), a power of two of lanes per row.
template <typename P, bool TO_SMEM>
__device__ __forceinline__ void move_rows(P* mem, P* sm, int n_rows, int words, int64_t pitch, int s_pitch) {
  int sh = 0;
  while ((1 << sh) < words && sh < 5) ++sh;
  const int lane = threadIdx.x & ((1 << sh) - 1);
  for (int r = threadIdx.x >> sh; r < n_rows; r += kOpsThreads >> sh)
    for (int w = lane; w < words; w += 1 << sh) {
      if (TO_SMEM) sm[r * s_pitch + w] = mem[r * pitch + w];
      else mem[r * pitch + w] = sm[r * s_pitch + w];
    }
}

template <typename E, bool TO_SMEM>
__device__ __forceinline__ void move_rows_of(E* mem, E* sm, int n_rows, int cn, int C, int stride) {
  constexpr int PER = sizeof(E) < 4 ? 4 / (int)sizeof(E) : 1;
  if (PER > 1 && cn % PER == 0 && C % PER == 0 && ((uintptr_t)mem & 3) == 0)
    move_rows<uint32_t, TO_SMEM>((uint32_t*)mem, (uint32_t*)sm, n_rows, cn / PER, C / PER, stride / PER);
  else
    move_rows<E, TO_SMEM>(mem, sm, n_rows, cn, C, stride);
}

// The first `cn` channels of consecutive rows to shared memory, asynchronously; false (nothing done) where they are not whole 4-byte
// words.
template <typename E>
__device__ __forceinline__ bool copy_rows_ahead(const E* mem, E* sm, int n_rows, int cn, int C, int stride) {
  if ((cn * sizeof(E) | C * sizeof(E) | (uintptr_t)mem) & 3u) return false;
  const int words = cn * (int)sizeof(E) / 4, pitch = C * (int)sizeof(E) / 4, s_pitch = stride * (int)sizeof(E) / 4;
  int sh = 0;
  while ((1 << sh) < words && sh < 5) ++sh;
  const int lane = threadIdx.x & ((1 << sh) - 1);
  const uint32_t to = (uint32_t)__cvta_generic_to_shared(sm);
  for (int r = threadIdx.x >> sh; r < n_rows; r += kOpsThreads >> sh)
    for (int w = lane; w < words; w += 1 << sh)
      asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(to + (uint32_t)(r * s_pitch + w) * 4u),
                   "l"((const uint32_t*)mem + (int64_t)r * pitch + w) : "memory");
  return true;
}

template <typename E, int V, bool BACK>
__global__ void __launch_bounds__(kOpsThreads)
dense_channels_first_kernel(E* __restrict__ rows, const int* __restrict__ z_idx, const int* __restrict__ z_ptr,
                            int64_t nnz, int64_t cols_per_b, int cols_per_block, int D, int C, int chunk, int stride,
                            E* __restrict__ dense, int* __restrict__ status) {
  after_previous<false>();
  extern __shared__ __align__(16) unsigned char smem[];
  int* s_map = (int*)smem;                                        // [cells] staged row of the cell or -1
  int* s_ptr = s_map + cols_per_block * D;                        // [columns + 1] first row of each column, and behind the last
  E* s_rows = (E*)(smem + ((size_t)(cols_per_block * (D + 1) + 1) * sizeof(int) + 15) / 16 * 16);   // [rows][stride]
  const int tid = threadIdx.x;
  const int64_t col0 = (int64_t)blockIdx.x * cols_per_block;
  const int nc = (int)min((int64_t)cols_per_block, cols_per_b - col0);
  const int64_t gcol0 = (int64_t)blockIdx.y * cols_per_b + col0;
  const int cells = nc * D;
  // Two round trips to memory before the first store: the columns' prefixes, then rows and depths together (they were five; 8 grids of
  // 131 k cells with 64 channels of fp16, a third of them filled: 58 -> 37 us).
  for (int i = tid; i <= nc; i += kOpsThreads) s_ptr[i] = i == 0 ? col_begin(z_ptr, gcol0) : __ldg(z_ptr + gcol0 + i - 1);
  for (int i = tid; i < cells; i += kOpsThreads) s_map[i] = -1;
  __syncthreads();
  const int64_t r0 = max((int64_t)0, min((int64_t)s_ptr[0], nnz));
  const int n_rows = (int)(min((int64_t)s_ptr[nc], nnz) - r0);
  const bool crowded = n_rows > cells;
  auto cell_of = [&](int i) {              // of row r0 + i, or -1
    int lo = 0, hi = nc - 1;               // first column of the block whose inclusive prefix exceeds the row
    while (lo < hi) {
      const int mid = (lo + hi) >> 1;
      if (s_ptr[mid + 1] > r0 + i) hi = mid; else lo = mid + 1;
    }
    const int z = __ldg(z_idx + r0 + i);
    return (unsigned)z < (unsigned)D ? lo * D + z : -1;
  };
  // rows of the first channels, on their way to shared memory while the map of the cells is made
  const bool ahead = !BACK && !crowded && copy_rows_ahead(rows + r0 * C, s_rows, n_rows, min(chunk, C), C, stride);
  bool others = false;                     // a row that does not own its cell
  for (int i = tid; i < n_rows; i += kOpsThreads) {
    const int cell = cell_of(i);
    if (cell < 0) {
      others = true;
      if (status) atomicOr(status, SPH_STATUS_BAD_INDEX);
    } else {
      others |= atomicMax(s_map + cell, i) >= 0;
    }
  }
  const int64_t vol = cols_per_b * D;
  E* plane0 = dense + (int64_t)blockIdx.y * C * vol + col0 * D;
  struct alignas(V * sizeof(E)) Vec { E e[V]; };
  constexpr int PAIR = sizeof(E) == 2 && V > 1 ? 2 : 1;
  if (BACK) others = __syncthreads_or(others);
  else if (crowded) __syncthreads();
  for (int c0 = 0; c0 < C; c0 += chunk) {
    const int cn = min(chunk, C - c0);
    E* mem = rows + r0 * C + c0;
    if (!BACK) {
      if (c0 == 0 && ahead) {
        asm volatile("cp.async.wait_all;" ::: "memory");
      } else if (!crowded) {
        move_rows_of<E, true>(mem, s_rows, n_rows, cn, C, stride);
      } else {
        for (int e = tid; e < cells * cn; e += kOpsThreads) {
          const int cell = e / cn, c = e % cn, r = s_map[cell];
          if (r >= 0) s_rows[cell * stride + c] = mem[(int64_t)r * C + c];
        }
      }
      __syncthreads();
    }
    // a thread keeps the staged rows of its V cells in registers and walks channels, two at a time for 2-byte elements
    // (one 4-byte access to shared memory per cell and pair)
    const int groups = cells / V;
    const int lanes = groups < kOpsThreads ? kOpsThreads / groups : 1;
    for (int t = tid; t < groups * lanes; t += kOpsThreads) {
      const int g = t % groups;
      int at[V];
#pragma unroll
      for (int j = 0; j < V; ++j) {
        const int r = s_map[g * V + j];
        at[j] = r < 0 ? -1 : (crowded ? g * V + j : r) * stride;
      }
      Vec* cell = (Vec*)(plane0 + (int64_t)c0 * vol) + g;
      const int64_t plane = vol / V;
      int c = t / groups * PAIR;
      for (; c + PAIR <= cn; c += lanes * PAIR) {
        Vec v[PAIR];
        if (BACK) {
#pragma unroll
          for (int q = 0; q < PAIR; ++q) v[q] = cell[(c + q) * plane];
#pragma unroll
          for (int j = 0; j < V; ++j)
            if (at[j] >= 0) {
              if constexpr (PAIR == 2) *(uint32_t*)(s_rows + at[j] + c) = (uint32_t)v[0].e[j] | (uint32_t)v[1].e[j] << 16;
              else s_rows[at[j] + c] = v[0].e[j];
            }
        } else {
#pragma unroll
          for (int j = 0; j < V; ++j) {
            if constexpr (PAIR == 2) {
              const uint32_t w = at[j] >= 0 ? *(const uint32_t*)(s_rows + at[j] + c) : 0u;
              v[0].e[j] = (E)w;
              v[1].e[j] = (E)(w >> 16);
            } else {
              v[0].e[j] = at[j] >= 0 ? s_rows[at[j] + c] : E(0);
            }
          }
#pragma unroll
          for (int q = 0; q < PAIR; ++q) cell[(c + q) * plane] = v[q];
        }
      }
      if (PAIR == 2 && c < cn) {          // the last of an odd number of channels
        Vec v;
        if (BACK) v = cell[c * plane];
#pragma unroll
        for (int j = 0; j < V; ++j) {
          if (!BACK) v.e[j] = at[j] >= 0 ? s_rows[at[j] + c] : E(0);
          else if (at[j] >= 0) s_rows[at[j] + c] = v.e[j];
        }
        if (!BACK) cell[c * plane] = v;
      }
    }
    __syncthreads();
    if (BACK) {
      if (!others) {
        move_rows_of<E, false>(mem, s_rows, n_rows, cn, C, stride);
      } else {
        for (int i = tid; i < n_rows; i += kOpsThreads) {
          const int cell = cell_of(i);
          const E* src = s_rows + (cell < 0 ? 0 : crowded ? cell : s_map[cell]) * stride;
          for (int c = 0; c < cn; ++c) mem[(int64_t)i * C + c] = cell < 0 ? E(0) : src[c];
        }
      }
      __syncthreads();
    }
  }
  if (BACK && blockIdx.x == gridDim.x - 1 && blockIdx.y == gridDim.y - 1)    // rows behind the last column's
    for (int64_t e = (r0 + max(n_rows, 0)) * C + tid; e < nnz * C; e += kOpsThreads) rows[e] = E(0);
}

template <typename E, int V>
int launch_dense_cf(void* rows, const int* z_idx, const int* z_ptr, int64_t nnz, int B, int64_t cols_per_b, int D, int C,
                    void* dense, int backward, int* status, cudaStream_t st) {
  int most = kDenseCells;
  while (most < kDenseMaxCells && (int64_t)2 * most * C * (int64_t)sizeof(E) <= kDenseBytes && B * cols_per_b * D >= 2 * most * kDenseBlocks)
    most *= 2;
  int cols = D >= most ? 1 : most / D;
  while (cols > 1 && (int64_t)cols * D % V) --cols;
  const int cells = cols * D;
  // as many channels at a time as fit in 64 KB when every cell holds a row; an odd number of 4-byte words per row, so that
  // consecutive rows start on other banks
  int chunk = (int)(65536 / ((int64_t)cells * sizeof(E)));
  chunk = chunk > C ? C : chunk < 1 ? 1 : chunk;
  constexpr int per = sizeof(E) < 4 ? 4 / (int)sizeof(E) : 1;
  const int stride = (div_up(chunk, per) | 1) * per;
  const int smem = ((cells + cols + 1) * (int)sizeof(int) + 15) / 16 * 16 + cells * stride * (int)sizeof(E);
  auto kern = backward ? dense_channels_first_kernel<E, V, true> : dense_channels_first_kernel<E, V, false>;
  SPH_CUDA(allow_smem(kern, kDenseSmem));
  launch(kern, dim3((unsigned)div_up64(cols_per_b, cols), (unsigned)B), kOpsThreads, smem, st, (E*)rows, z_idx, z_ptr, nnz, cols_per_b, cols, D, C, chunk, stride, (E*)dense, status);
  SPH_LAUNCH_CHECK();
  return SPH_OK;
}

template <typename E>
int dense_cf(void* rows, const int* z_idx, const int* z_ptr, int64_t nnz, int B, int64_t cols_per_b, int D, int C,
             void* dense, int backward, int* status, cudaStream_t st) {
  // 16-byte vectors where every channel plane and every block of columns starts on one
  constexpr int V = 16 / (int)sizeof(E);
  if (cols_per_b * D % V == 0 && D % V == 0 && ((uintptr_t)dense & 15) == 0)
    return launch_dense_cf<E, V>(rows, z_idx, z_ptr, nnz, B, cols_per_b, D, C, dense, backward, status, st);
  return launch_dense_cf<E, 1>(rows, z_idx, z_ptr, nnz, B, cols_per_b, D, C, dense, backward, status, st);
}

int piece_bytes(int row_bytes, const void* a, const void* b) {
  const uintptr_t bits = (uintptr_t)a | (uintptr_t)b | (uintptr_t)row_bytes;
  if ((bits & 15) == 0) return 16;
  if ((bits & 3) == 0) return 4;
  if ((bits & 1) == 0) return 2;
  return 1;
}

struct InitScratch {
  int words;
  int64_t ncols;
  size_t mask_bytes, blocksum_bytes;
};
InitScratch init_layout(int B, const int32_t shape[3]) {
  InitScratch l;
  l.words = div_up(shape[2], 32);
  l.ncols = (int64_t)B * shape[0] * shape[1];
  l.mask_bytes = ((size_t)l.ncols * l.words * sizeof(uint32_t) + 255) & ~(size_t)255;
  l.blocksum_bytes = ((size_t)div_up64(l.ncols, 256) * sizeof(int) + 255) & ~(size_t)255;
  return l;
}

}  // namespace

}  // namespace sph

using namespace sph;

extern "C" int64_t sph_init_tensor_scratch_bytes(int32_t B, const int32_t shape[3]) {
  if (B <= 0 || !shape || shape[0] <= 0 || shape[1] <= 0 || shape[2] <= 0) return SPH_ERR_INVALID;
  const InitScratch l = init_layout(B, shape);
  return (int64_t)(256 + l.mask_bytes + l.blocksum_bytes);
}

extern "C" int sph_init_tensor(const void* d_feature, int32_t row_bytes, int64_t nnz, const int32_t* d_indices,
                               int32_t B, const int32_t shape[3], void* d_scratch, void* d_out_feature,
                               int32_t* d_z_idx, int32_t* d_z_ptr, int32_t* d_permutation, int32_t* d_status,
                               void* stream) {
  SPH_CHECK_ARG(B > 0 && shape && shape[0] > 0 && shape[1] > 0 && shape[2] > 0, "batch and shape must be positive");
  SPH_CHECK_ARG(nnz >= 0 && row_bytes >= 0 && nnz < 0x7fffffffLL, "bad sizes");
  SPH_CHECK_ARG(d_scratch && d_z_ptr, "null pointer");
  SPH_CHECK_ARG(nnz == 0 || (d_indices && d_z_idx && d_permutation && (row_bytes == 0 || (d_feature && d_out_feature))),
                "null pointer");
  SPH_CHECK_ARG(((uintptr_t)d_indices & 15) == 0, "indices must be 16-byte aligned");
  const InitScratch l = init_layout(B, shape);
  SPH_CHECK_ARG(l.ncols <= 0x7fffffffLL, "more than 2^31 columns");
  cudaStream_t st = (cudaStream_t)stream;
  int* header = (int*)d_scratch;                           // [0] = total
  uint32_t* mask = (uint32_t*)((char*)d_scratch + 256);
  int* blocksum = (int*)((char*)d_scratch + 256 + l.mask_bytes);
  SPH_CUDA(cudaMemsetAsync(d_scratch, 0, 256 + l.mask_bytes, st));
  const int H = shape[0], W = shape[1], D = shape[2];
  if (nnz > 0) {
    launch(mark_voxels_kernel, (unsigned)div_up64(nnz, kOpsThreads), kOpsThreads, 0, st, d_indices, nnz, B, H, W, D, l.words,
                                                                                      mask, d_status);
    SPH_LAUNCH_CHECK();
  }
  int rc = column_prefix_from_masks(mask, l.words, l.ncols, d_z_ptr, blocksum, header, nullptr, st);
  if (rc != SPH_OK) return rc;
  if (nnz > 0) {
    launch(place_voxels_kernel, (unsigned)div_up64(nnz, kOpsThreads), kOpsThreads, 0, st, d_indices, nnz, B, H, W, D, l.words,
                                                                                       mask, d_z_ptr, d_z_idx,
                                                                                       d_permutation);
    SPH_LAUNCH_CHECK();
    if (row_bytes > 0) {
      rc = sph_permute_rows(d_feature, row_bytes, nnz, d_permutation, 0, d_out_feature, stream);
      if (rc != SPH_OK) return rc;
    }
  }
  return SPH_OK;
}

extern "C" int sph_permute_rows(const void* d_src, int32_t row_bytes, int64_t n_rows, const int32_t* d_permutation,
                                int gather, void* d_dst, void* stream) {
  SPH_CHECK_ARG(n_rows >= 0 && row_bytes >= 0, "bad sizes");
  if (n_rows == 0 || row_bytes == 0) return SPH_OK;
  SPH_CHECK_ARG(d_src && d_dst && d_permutation, "null pointer");
  cudaStream_t st = (cudaStream_t)stream;
  const int pb = piece_bytes(row_bytes, d_src, d_dst);
  const int pieces = row_bytes / pb;
  const unsigned blocks = (unsigned)div_up64(n_rows * pieces, kOpsThreads);
  switch (pb) {
    case 16: launch(permute_rows_kernel<uint4>, blocks, kOpsThreads, 0, st, (const uint4*)d_src, (uint4*)d_dst, d_permutation, n_rows, pieces, gather); break;
    case 4: launch(permute_rows_kernel<uint32_t>, blocks, kOpsThreads, 0, st, (const uint32_t*)d_src, (uint32_t*)d_dst, d_permutation, n_rows, pieces, gather); break;
    case 2: launch(permute_rows_kernel<uint16_t>, blocks, kOpsThreads, 0, st, (const uint16_t*)d_src, (uint16_t*)d_dst, d_permutation, n_rows, pieces, gather); break;
    default: launch(permute_rows_kernel<uint8_t>, blocks, kOpsThreads, 0, st, (const uint8_t*)d_src, (uint8_t*)d_dst, d_permutation, n_rows, pieces, gather); break;
  }
  SPH_LAUNCH_CHECK();
  return SPH_OK;
}

extern "C" int sph_to_dense(void* d_rows, int32_t row_bytes, int64_t nnz, const int32_t* d_z_idx,
                            const int32_t* d_z_ptr, int32_t B, const int32_t shape[3], void* d_dense, int backward,
                            int32_t* d_status, void* stream) {
  SPH_CHECK_ARG(B > 0 && shape && shape[0] > 0 && shape[1] > 0 && shape[2] > 0, "batch and shape must be positive");
  SPH_CHECK_ARG(nnz >= 0 && row_bytes >= 0, "bad sizes");
  if (nnz == 0 || row_bytes == 0) return SPH_OK;
  SPH_CHECK_ARG(d_rows && d_z_idx && d_z_ptr && d_dense, "null pointer");
  cudaStream_t st = (cudaStream_t)stream;
  const int64_t ncols = (int64_t)B * shape[0] * shape[1];
  const int pb = piece_bytes(row_bytes, d_rows, d_dense);
  const int pieces = row_bytes / pb;
  const unsigned blocks = (unsigned)div_up64(nnz * pieces, kOpsThreads);
  switch (pb) {
    case 16: launch(dense_rows_kernel<uint4>, blocks, kOpsThreads, 0, st, (uint4*)d_rows, d_z_idx, d_z_ptr, nnz, ncols, shape[2], pieces, (uint4*)d_dense, backward, d_status); break;
    case 4: launch(dense_rows_kernel<uint32_t>, blocks, kOpsThreads, 0, st, (uint32_t*)d_rows, d_z_idx, d_z_ptr, nnz, ncols, shape[2], pieces, (uint32_t*)d_dense, backward, d_status); break;
    case 2: launch(dense_rows_kernel<uint16_t>, blocks, kOpsThreads, 0, st, (uint16_t*)d_rows, d_z_idx, d_z_ptr, nnz, ncols, shape[2], pieces, (uint16_t*)d_dense, backward, d_status); break;
    default: launch(dense_rows_kernel<uint8_t>, blocks, kOpsThreads, 0, st, (uint8_t*)d_rows, d_z_idx, d_z_ptr, nnz, ncols, shape[2], pieces, (uint8_t*)d_dense, backward, d_status); break;
  }
  SPH_LAUNCH_CHECK();
  return SPH_OK;
}

extern "C" int sph_dense_channels_first(void* d_rows, int32_t elem_bytes, int32_t channels, int64_t nnz,
                                        const int32_t* d_z_idx, const int32_t* d_z_ptr, int32_t B, const int32_t shape[3],
                                        void* d_dense, int backward, int32_t* d_status, void* stream) {
  SPH_CHECK_ARG(B > 0 && B <= 65535 && shape && shape[0] > 0 && shape[1] > 0 && shape[2] > 0,
                "batch and shape must be positive");
  SPH_CHECK_ARG(nnz >= 0 && channels > 0, "bad sizes");
  SPH_CHECK_ARG(d_z_ptr && d_dense && (nnz == 0 || (d_rows && d_z_idx)), "null pointer");
  if (shape[2] > kDenseMaxCells) {
    set_error("sph_dense_channels_first: columns of more than %d cells are not supported", kDenseMaxCells);
    return SPH_ERR_LIMIT;
  }
  const int64_t cols = (int64_t)shape[0] * shape[1];
  cudaStream_t st = (cudaStream_t)stream;
  switch (elem_bytes) {
    case 1: return dense_cf<uint8_t>(d_rows, d_z_idx, d_z_ptr, nnz, B, cols, shape[2], channels, d_dense, backward, d_status, st);
    case 2: return dense_cf<uint16_t>(d_rows, d_z_idx, d_z_ptr, nnz, B, cols, shape[2], channels, d_dense, backward, d_status, st);
    case 4: return dense_cf<uint32_t>(d_rows, d_z_idx, d_z_ptr, nnz, B, cols, shape[2], channels, d_dense, backward, d_status, st);
    case 8: return dense_cf<uint64_t>(d_rows, d_z_idx, d_z_ptr, nnz, B, cols, shape[2], channels, d_dense, backward, d_status, st);
  }
  set_error("sph_dense_channels_first: elements of %d bytes", elem_bytes);
  return SPH_ERR_UNSUPPORTED;
}

// ---- backward of the fused epilogue relu(acc + bias): gradient mask and bias gradient in one pass ---------------
namespace sph {
namespace {

__device__ __forceinline__ float ld_f(const float* p, int64_t i) { return p[i]; }
__device__ __forceinline__ float ld_f(const __half* p, int64_t i) { return __half2float(p[i]); }
__device__ __forceinline__ float ld_f(const __nv_bfloat16* p, int64_t i) { return __bfloat162float(p[i]); }
__device__ __forceinline__ void st_f(float* p, int64_t i, float v) { p[i] = v; }
__device__ __forceinline__ void st_f(__half* p, int64_t i, float v) { p[i] = __float2half_rn(v); }
__device__ __forceinline__ void st_f(__nv_bfloat16* p, int64_t i, float v) { p[i] = __float2bfloat16_rn(v); }

constexpr int kEpiThreads = 256;

// d_pre[r][c] = out[r][c] > 0 ? d_out[r][c] : 0 (relu) or d_out (no relu); d_bias[c] += sum_r d_pre[r][c].
// A thread stays on one channel (the first floor(256 / C) * C threads of a block work, the rest only join the
// barrier), walks rows with a grid stride and keeps its sum in a register; sums of equal channels meet in shared
// memory, one atomic per channel and block.
template <typename T>
__global__ void __launch_bounds__(kEpiThreads)
epilogue_backward_kernel(const T* __restrict__ d_out, const T* __restrict__ out, int64_t n, int C, int relu,
                         T* __restrict__ d_pre, float* __restrict__ d_bias) {
  after_previous();
  __shared__ float s_sum[kEpiThreads];
  const int c = threadIdx.x % C;
  const int rows_per_block = kEpiThreads / C;
  const int active = rows_per_block * C;
  float sum = 0.f;
  for (int64_t r = (int64_t)blockIdx.x * rows_per_block + threadIdx.x / C; r < n && (int)threadIdx.x < active;
       r += (int64_t)gridDim.x * rows_per_block) {
    const int64_t i = r * C + c;
    float g = ld_f(d_out, i);
    if (relu && !(ld_f(out, i) > 0.f)) g = 0.f;
    if (d_pre) st_f(d_pre, i, g);
    sum += g;
  }
  if (d_bias) {
    s_sum[threadIdx.x] = sum;
    __syncthreads();
    if (threadIdx.x < C) {
      float t = 0.f;
      for (int j = threadIdx.x; j < active; j += C) t += s_sum[j];
      atomicAdd(d_bias + threadIdx.x, t);
    }
  }
}

// The same with 16-byte loads and stores (channels a multiple of the V elements of one): a thread owns one vector of
// channels, keeps V sums and has kVecRows rows in flight.  Bound by memory: 1.39 M rows of 64 bf16 channels (534 MB)
// 194 -> 84 us.
constexpr int kVecRows = 4;

template <typename T>
__global__ void __launch_bounds__(kEpiThreads)
epilogue_backward_vec_kernel(const T* __restrict__ d_out, const T* __restrict__ out, int64_t n, int C, int relu,
                             T* __restrict__ d_pre, float* __restrict__ d_bias) {
  after_previous();
  constexpr int V = 16 / (int)sizeof(T);
  struct alignas(16) Vec { T e[V]; };
  __shared__ float s_sum[kEpiThreads];                 // [C], C <= 256
  const int per = C / V;                               // vectors of a row; threads beyond rows x per idle
  const int rows_per_block = kEpiThreads / per;
  const int c = threadIdx.x % per, r_in = threadIdx.x / per;
  float sum[V];
#pragma unroll
  for (int j = 0; j < V; ++j) sum[j] = 0.f;
  for (int i = threadIdx.x; i < C; i += kEpiThreads) s_sum[i] = 0.f;
  __syncthreads();
  const int64_t stride = (int64_t)gridDim.x * rows_per_block;
  if (r_in < rows_per_block) {
    for (int64_t r = (int64_t)blockIdx.x * rows_per_block + r_in; r < n; r += stride * kVecRows) {
      Vec g[kVecRows], o[kVecRows];
#pragma unroll
      for (int u = 0; u < kVecRows; ++u) {
        const int64_t at = (r + u * stride) * per + c;
        if (r + u * stride < n) {
          g[u] = ((const Vec*)d_out)[at];
          if (relu) o[u] = ((const Vec*)out)[at];
        }
      }
#pragma unroll
      for (int u = 0; u < kVecRows; ++u) {
        if (r + u * stride >= n) continue;
#pragma unroll
        for (int j = 0; j < V; ++j) {
          if (relu && !(ld_f(o[u].e, j) > 0.f)) st_f(g[u].e, j, 0.f);
          sum[j] += ld_f(g[u].e, j);
        }
        if (d_pre) ((Vec*)d_pre)[(r + u * stride) * per + c] = g[u];
      }
    }
  }
  if (d_bias) {
    // lanes of equal channels first (per divides the warp), then the warps
    if (32 % per == 0) {
#pragma unroll
      for (int j = 0; j < V; ++j)
        for (int o = per; o < 32; o <<= 1) sum[j] += __shfl_xor_sync(0xffffffffu, sum[j], o);
      if ((threadIdx.x & 31) >= per) goto counted;
    }
    if (r_in < rows_per_block)
#pragma unroll
      for (int j = 0; j < V; ++j) atomicAdd(s_sum + c * V + j, sum[j]);
  counted:
    __syncthreads();
    for (int i = threadIdx.x; i < C; i += kEpiThreads) atomicAdd(d_bias + i, s_sum[i]);
  }
}

template <typename T>
bool launch_epilogue_vec(const void* d_out, const void* out, int64_t n, int C, int relu, void* d_pre, float* d_bias, cudaStream_t st) {
  constexpr int V = 16 / (int)sizeof(T);
  if (C % V != 0 || (((uintptr_t)d_out | (uintptr_t)out | (uintptr_t)d_pre) & 15) != 0) return false;
  const int rows_per_block = kEpiThreads / (C / V);
  int64_t blocks = div_up64(n, (int64_t)rows_per_block * kVecRows);
  const int sms = current_sm_count();
  if (blocks > (int64_t)sms * 8) blocks = (int64_t)sms * 8;
  launch(epilogue_backward_vec_kernel<T>, (unsigned)blocks, kEpiThreads, 0, st, (const T*)d_out, (const T*)out, n, C, relu, (T*)d_pre, d_bias);
  return true;
}

}  // namespace
}  // namespace sph

extern "C" int sph_epilogue_backward(const void* d_dout, const void* d_out, int dtype, int64_t n, int32_t channels,
                                     int relu, void* d_dpre, float* d_dbias, void* stream) {
  SPH_CHECK_ARG(n >= 0 && channels > 0, "bad sizes");
  SPH_CHECK_ARG(dtype == SPH_F32 || dtype == SPH_F16 || dtype == SPH_BF16, "unsupported dtype");
  SPH_CHECK_ARG(channels <= kEpiThreads, "at most 256 channels");
  cudaStream_t st = (cudaStream_t)stream;
  if (d_dbias) SPH_CUDA(cudaMemsetAsync(d_dbias, 0, (size_t)channels * sizeof(float), st));
  if (n == 0) return SPH_OK;
  SPH_CHECK_ARG(d_dout && (!relu || d_out) && (d_dpre || d_dbias), "null pointer");
  const bool vec = dtype == SPH_F32   ? launch_epilogue_vec<float>(d_dout, d_out, n, channels, relu, d_dpre, d_dbias, st)
                   : dtype == SPH_F16 ? launch_epilogue_vec<__half>(d_dout, d_out, n, channels, relu, d_dpre, d_dbias, st)
                                      : launch_epilogue_vec<__nv_bfloat16>(d_dout, d_out, n, channels, relu, d_dpre, d_dbias, st);
  if (vec) {
    SPH_LAUNCH_CHECK();
    return SPH_OK;
  }
  const int rows_per_block = kEpiThreads / channels;
  int64_t blocks = div_up64(n, (int64_t)rows_per_block * 8);      // ~8 rows per thread
  if (blocks > 148 * 16) blocks = 148 * 16;
  if (blocks < 1) blocks = 1;
  switch (dtype) {
    case SPH_F32: launch(epilogue_backward_kernel<float>, (unsigned)blocks, kEpiThreads, 0, st, (const float*)d_dout, (const float*)d_out, n, channels, relu, (float*)d_dpre, d_dbias); break;
    case SPH_F16: launch(epilogue_backward_kernel<__half>, (unsigned)blocks, kEpiThreads, 0, st, (const __half*)d_dout, (const __half*)d_out, n, channels, relu, (__half*)d_dpre, d_dbias); break;
    default: launch(epilogue_backward_kernel<__nv_bfloat16>, (unsigned)blocks, kEpiThreads, 0, st, (const __nv_bfloat16*)d_dout, (const __nv_bfloat16*)d_out, n, channels, relu, (__nv_bfloat16*)d_dpre, d_dbias); break;
  }
  SPH_LAUNCH_CHECK();
  return SPH_OK;
}
