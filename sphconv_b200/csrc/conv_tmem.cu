// Output-stationary gather-GEMM on the Blackwell tensor cores (tcgen05) with the gathered rows in tensor memory.
//
//   out[r,:] = epilogue( sum_k rows[nbr[k][r], :] @ W[k] )          r in [0, n_out), 9 or 27 offsets
//
//   D[128 rows x oC] += X_k[128 x iC] * W[k][iC x oC]
//   A operand = 128 gathered neighbour rows of offset k, in TMEM (lane = output row);
//   B operand = W[k]^T, N = oC, K-major, pre-packed once per weight (the image conv_tc.cu uses as its A operand);
//   D         = fp32 / int32 accumulator in TMEM, lane = output row, column = output channel.
//
// Rows are numbered along the columns of the grid, so the neighbours that consecutive output rows have in one line of
// columns - a third of the offsets: those of one kernel height - lie in one short run of consecutive input rows.  TMA brings
// that run to shared memory once per tile and line (tensor map with the swizzle of the row width, any number of 32-row boxes);
// for every offset each lane then reads the row of ITS neighbour with 16-byte loads and writes it to the TMEM lane of its
// output row.  Against gathering every pair's row into the UMMA core-matrix layout with cp.async (conv_tc.cu, conv_tc_rows.cu)
//  * a row is copied to shared memory 3 times a tile instead of up to 27 times, by TMA instead of by lanes;
//  * the multiplication reads only the weights from shared memory;
//  * the operand is handed over by 4 arrivals of warps instead of 128 of threads.
// The order of sums is that of the other tensor-core kernels (offsets ascending, 32 bytes of a row per instruction), and so are
// the results, bit for bit.  Measured against them (us, L2 flushed; tables of 27 offsets, share of neighbours present):
//   32 -> 32 fp16, 1.5 M rows, 0.44   328 -> 201      64 -> 64 fp16, 683 k rows, 0.82   253 -> 172
//   16 -> 32 fp16, 1.5 M rows, 0.05   200 -> 170      64 -> 32 fp16, 1.5 M rows, 0.12   515 -> 195
//   32 -> 32 int8, 1.5 M rows, 0.44   255 -> 168      64 -> 64 fp16,  22 k rows, 0.69  25.6 -> 22.5
// Bound by no single unit: issue slots 75, 71 and 61 % busy at 32-, 64- and 128-byte rows, the shared-memory data path
// 41, 71 and 68 % (786 k rows of 16 -> 32 and 32 -> 32, 347 k of 64 -> 64); without the TMEM writes and the loads in front of them a
// 32 -> 32 layer takes 141 instead of 206 us.  Tried and
// slower: entries kept in registers with the offsets unrolled (instruction fetch: 577); rows of zeros in shared memory for absent
// neighbours (bank conflicts: 263); the instruction's disable-output-lane mask instead of zeros (its operands: 217).
//
// A run longer than its buffer (tiles that pass from one line of columns into the next, dense or deep columns, strides that thin
// the output, tables without locality) is read around it: the gather takes the table's entries a batch ahead, rows inside the
// buffer from there and the others straight into registers, 32 bytes a load.  Against asking the table offset by offset when a
// row was found missing (us, launches one behind the other): 32 -> 64 strided, 146 k rows of surfaces, 91 % of the lines too long,
// 59 -> 38; 16 -> 32 strided, 111 k rows, 9 % too long, 30 -> 22; input gradient 32 -> 16, 284 k rows, 77 % too long, 82 -> 51;
// 32 -> 32 without locality, 300 k rows, 119 -> 78.  Bound there by the latency of L2: a warp has one batch in flight.  Both kinds
// of line in one loop are slower (the state of one costs the other: 3 % over 130 tables, 32 -> 32 on 1.5 M rows 201 against 194).
//
// A CTA owns 256 consecutive output rows at a time (two halves of M = 128; one half where the tiles would not fill the SMs)
// and is persistent over such tiles.  Warp roles: 0-15 gather (warp w: TMEM lanes 32 (w % 4) of half w / 4 % 2, and the batches
// of offsets of team w / 8), 16 and 17 issue the MMAs of a half each, 18-21 run the epilogue, 22 issues the TMA loads of the
// runs, 23 those of the weight images, 24-31 plan.
//  * The planning warps run up to two tiles ahead: they read the table entries of their 32 rows, find the run of each line and
//    the offsets that occur in each half, and leave for the gather warps where in its run the neighbour of each row lies (16
//    bits), offset after offset that occurs.  Any table is right, also one whose runs the buffers do not hold.
//  * Offsets that no row of a half has are skipped (half of them in the input gradient of a strided layer); a row without a
//    neighbour at an offset that others have brings zeros, without an access to shared memory.
//  * Every wait is made by a whole warp and MMAs are issued by an elected lane in converged code: an MMA from a divergent
//    branch takes 57 to 125 cycles to issue (its operands are moved to uniform registers one by one) and 16 to 32 from converged
//    code, which is what the tensor pipe needs for M = 128, N = 32 to 64; a barrier that is ready costs 300 cycles to
//    wait for in a branch of one lane and 60 to 80 in converged code.
#include <cuda.h>

#include "common.cuh"
#include "tc_common.cuh"

namespace sph {

#ifdef SPH_TEST_HOOKS
extern int g_test_withhold;         // conv_tc.cu
#endif

namespace {
namespace tmemform {

using namespace tc;

constexpr int kThreads = 1024;
constexpr int kHalfRows = 128;
constexpr int kMmaWarp = 16, kEpiWarp = 18, kRunWarp = 22, kWeightWarp = 23, kPlanWarp = 24;
constexpr int kTeams = 2;             // gather warps of a TMEM lane quarter: they take alternate batches
constexpr int kLines = 3;             // groups of offsets that share a run
constexpr int kRunSlots = 3;          // most runs in shared memory (plan_smem)
constexpr int kBox = 32;              // rows a TMA load brings
constexpr int kOperandCols = 32;      // TMEM columns of an operand: one batch of one to four offsets
constexpr int kOperands = 4;          // operands of a half in TMEM
constexpr int kWeightSlots = 8;       // most streamed weight images in flight (plan_smem)
constexpr uint32_t kScattered = 64;   // a run of this many times the rows that a slot holds is not brought (8: 200 instead of 192 us)
constexpr uint32_t kAbsent = 0xffffu;   // place of a neighbour that there is not
constexpr int kStagePieces = 8;       // 16-byte pieces of the widest output row that is staged (the narrowest: half as many)
constexpr int kSmemTotal = 227 * 1024 - 2048;   // dynamic shared memory available next to the static part

struct Partial {                      // what a planning warp found, for the others
  int2 run[kLines];                   // smallest (as unsigned) and largest entry of a line
  uint32_t offsets;                   // offsets that any of its rows has
  uint32_t unused;
};
struct __align__(16) Plan {
  uint32_t lo[kLines];                // first row of a line's run
  uint32_t offsets0;                  // offsets of half 0, of half 1
  int hi[kLines];                     // its last row, -1: no entry in the line
  uint32_t offsets1;
};

struct TmemParams {
  const void* rows;
  const void* packed;                 // [KV] images of W[k]^T, each N x K_ch, K-major
  const int* nbr;                     // [KV][n_out]
  int64_t n_rows, n_out;
  int N, flip_k;
  int halves, num_tiles;
  int w_bytes;
  int weight_slots;                   // streamed weight images in flight
  int run_slots;                      // runs in shared memory
  int cap;                            // rows of a run that a slot holds, a multiple of kBox
  int plan_off, part_off, epi_off, place_off, w_off, run_off;   // from the 1024-byte-aligned base
  int stage_off;                      // -1: output rows are not staged
  int is_bf16;
  const float* scale;
  Bias bias;
  int relu;
  void* out;
  int out_dtype, out_esize;
  int* status;
#ifdef SPH_TEST_HOOKS
  int test_withhold;
#endif
};

// A operand of the instruction in TMEM (K-major: 16-bit elements two to a column, 8-bit elements four).
template <bool I8>
__device__ __forceinline__ void umma_ta(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t acc) {
  if constexpr (I8)
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::i8 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(acc));
  else
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(acc));
}

// 32 consecutive columns of this thread's TMEM lane.
__device__ __forceinline__ void tmem_st_batch(uint32_t taddr, const uint4 (&v)[8]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,"
      "%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};" ::"r"(taddr),
      "r"(v[0].x), "r"(v[0].y), "r"(v[0].z), "r"(v[0].w), "r"(v[1].x), "r"(v[1].y), "r"(v[1].z), "r"(v[1].w), "r"(v[2].x),
      "r"(v[2].y), "r"(v[2].z), "r"(v[2].w), "r"(v[3].x), "r"(v[3].y), "r"(v[3].z), "r"(v[3].w), "r"(v[4].x), "r"(v[4].y),
      "r"(v[4].z), "r"(v[4].w), "r"(v[5].x), "r"(v[5].y), "r"(v[5].z), "r"(v[5].w), "r"(v[6].x), "r"(v[6].y), "r"(v[6].z),
      "r"(v[6].w), "r"(v[7].x), "r"(v[7].y), "r"(v[7].z), "r"(v[7].w)
      : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

__device__ __forceinline__ void tma_rows(uint32_t dst, const CUtensorMap* map, int row, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst),
      "l"(map), "r"(0), "r"(row), "r"(bar)
      : "memory");
}

// 16 bytes of shared memory where `present`, else zeros without an access (which would take its turn on the banks).
__device__ __forceinline__ uint4 lds128(uint32_t addr, bool present) {
  uint4 v = make_uint4(0u, 0u, 0u, 0u);
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %5, 0;\n\t@p ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];\n\t}"
               : "+r"(v.x), "+r"(v.y), "+r"(v.z), "+r"(v.w)
               : "r"(addr), "r"((int)present));
  return v;
}

// 32 bytes of global memory (as two pieces where the address is no multiple of 32) where `present`, else what a and b hold.
__device__ __forceinline__ void ldg256(uint4& a, uint4& b, const void* at, bool present, bool whole) {
  if (whole)
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %9, 0;\n\t@p ld.global.nc.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];\n\t}"
                 : "+r"(a.x), "+r"(a.y), "+r"(a.z), "+r"(a.w), "+r"(b.x), "+r"(b.y), "+r"(b.z), "+r"(b.w)
                 : "l"(at), "r"((int)present));
  else
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %9, 0;\n\t@p ld.global.nc.v4.b32 {%0,%1,%2,%3}, [%8];\n\t"
        "@p ld.global.nc.v4.b32 {%4,%5,%6,%7}, [%8 + 16];\n\t}"
        : "+r"(a.x), "+r"(a.y), "+r"(a.z), "+r"(a.w), "+r"(b.x), "+r"(b.y), "+r"(b.z), "+r"(b.w)
        : "l"(at), "r"((int)present));
}

// Byte offset of 16-byte piece 0 of row i in a run of KC-piece rows as TMA swizzles it (piece c: xor with 16 c).
template <int KC>
__device__ __forceinline__ uint32_t row_at(uint32_t i) {
  const uint32_t x = KC == 8 ? i & 7u : KC == 4 ? (i >> 1) & 3u : (i >> 2) & 1u;
  return i * (KC * 16u) + (x << 4);
}

// The runs of a tile and the offsets its halves have, from what the planning warps found; called by whole warps.
__device__ __forceinline__ Plan combine(const Partial* part, int lane) {
  uint32_t lo = ~0u, bits = 0u;
  int hi = -1;
  if (lane < 8 * kLines) {
    const int2 v = part[lane & 7].run[lane >> 3];
    lo = (uint32_t)v.x;
    hi = v.y;
  } else {
    bits = part[lane - 8 * kLines].offsets;
  }
  Plan r;
#pragma unroll
  for (int l = 0; l < kLines; ++l) {
    r.lo[l] = __reduce_min_sync(0xffffffffu, (lane >> 3) == l ? lo : ~0u);
    r.hi[l] = __reduce_max_sync(0xffffffffu, (lane >> 3) == l ? hi : -1);
  }
  // a half without any pair multiplies zeros once: its accumulator has to be written
  r.offsets0 = max(__reduce_or_sync(0xffffffffu, lane < 28 ? bits : 0u), 1u);
  r.offsets1 = max(__reduce_or_sync(0xffffffffu, lane < 28 ? 0u : bits), 1u);
  // a tile without any pair still brings a row, so that the gather never gets a tile ahead of the warp that issues the loads
  if ((r.hi[0] & r.hi[1] & r.hi[2]) < 0) {
    r.lo[0] = 0u;
    r.hi[0] = 0;
  }
  return r;
}

// Rows of a run longer than `cap` that are brought to shared memory: its first ones, or none where the entries are scattered so
// widely that few of them would be among these.
__device__ __forceinline__ uint32_t held_of_split(uint32_t lo, int hi, uint32_t cap) {
  return ((uint32_t)hi - lo) / kScattered >= cap ? 0u : cap;
}

// 16 accumulator values of one output row (channels c0 .. c0+15) -> 16-byte pieces; returns how many.
template <bool I8>
__device__ __forceinline__ int convert16(uint4 (&to)[4], int out_dtype, const uint32_t (&raw)[16], const float* sc, const float* bi,
                                         int relu) {
  float x[16];
#pragma unroll
  for (int j = 0; j < 16; ++j) {
    float v = I8 ? (float)(int)raw[j] : __uint_as_float(raw[j]);
    v = fmaf(v, sc[j], bi[j]);
    x[j] = relu ? fmaxf(v, 0.f) : v;
  }
  if (out_dtype == SPH_F32) {
#pragma unroll
    for (int j = 0; j < 4; ++j)
      to[j] = make_uint4(__float_as_uint(x[4 * j]), __float_as_uint(x[4 * j + 1]), __float_as_uint(x[4 * j + 2]), __float_as_uint(x[4 * j + 3]));
    return 4;
  }
  if (out_dtype == SPH_I8) {
    uint32_t w[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      uint32_t acc = 0;
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        const int q = (int)fminf(fmaxf(rintf(x[4 * j + t]), -127.f), 127.f);
        acc |= ((uint32_t)q & 0xffu) << (8 * t);
      }
      w[j] = acc;
    }
    to[0] = make_uint4(w[0], w[1], w[2], w[3]);
    return 1;
  }
  uint32_t h[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    if (out_dtype == SPH_F16) {
      const __half2 v = __floats2half2_rn(x[2 * j], x[2 * j + 1]);
      h[j] = *(const uint32_t*)&v;
    } else {
      const __nv_bfloat162 v = __floats2bfloat162_rn(x[2 * j], x[2 * j + 1]);
      h[j] = *(const uint32_t*)&v;
    }
  }
  to[0] = make_uint4(h[0], h[1], h[2], h[3]);
  to[1] = make_uint4(h[4], h[5], h[6], h[7]);
  return 2;
}

// KC = 16-byte pieces of a row (2, 4, 8), I8 = int8 operands, L = offsets that share a run (9 of 27, 3 of 9).
template <int KC, bool I8, int L>
__global__ void __launch_bounds__(kThreads, 1) conv_gather_tmem_kernel(const __grid_constant__ CUtensorMap map, const TmemParams p) {
  constexpr int KV = kLines * L;
  constexpr int U = 8 / KC;                         // offsets of a batch
  constexpr int LP = (L + U - 1) / U * U;           // a line's list of places, in whole batches
  constexpr int ROW = KC * 16;
  constexpr bool STREAM = KC == 8;                  // weight images come offset by offset (else all stay in shared memory)
  extern __shared__ uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t s_run_full[kRunSlots], s_run_empty[kRunSlots];
  __shared__ __align__(8) uint64_t s_a_full[2][kOperands], s_a_empty[2][kOperands];
  __shared__ __align__(8) uint64_t s_w_full[kWeightSlots], s_w_empty[kWeightSlots];
  __shared__ __align__(8) uint64_t s_acc_full[2][2], s_acc_empty[2][2];   // [buffer][half]
  __shared__ __align__(8) uint64_t s_part[2], s_place_full[2], s_place_empty[2];
  __shared__ uint32_t s_tmem_base;
  __shared__ int s_abort;

  const int tid = threadIdx.x, lane = tid & 31;
  const int warp = (int)uniform((uint32_t)tid >> 5);
  const uint32_t base_u = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* base = smem_raw + (base_u - smem_u32(smem_raw));
  Plan* s_plan = (Plan*)(base + p.plan_off);        // [2]
  Partial* s_partial = (Partial*)(base + p.part_off);   // [2][8]
  float* s_epi = (float*)(base + p.epi_off);        // [2][64]: scale, bias of the epilogue
  uint16_t* s_place = (uint16_t*)(base + p.place_off);  // [2][8 warps][kLines * LP][32]: of neighbours, in 16 bytes from the start of the run
  const int halves = p.halves;

  const uint32_t cap = (uint32_t)p.cap;
  const uint32_t slot_bytes = cap * ROW;
  if (tid < 16) {
    for (int l = 0; l < kLines; ++l) s_partial[tid].run[l] = make_int2(-1, -1);
    s_partial[tid].offsets = 0u;
  }
  if (tid == 0) {
    s_abort = 0;
    for (int s = 0; s < p.run_slots; ++s) {
      mbar_init(smem_u32(&s_run_full[s]), 1);
      mbar_init(smem_u32(&s_run_empty[s]), 4 * kTeams * halves);
    }
    for (int h = 0; h < 2; ++h)
      for (int s = 0; s < kOperands; ++s) {
        mbar_init(smem_u32(&s_a_full[h][s]), 4);
        mbar_init(smem_u32(&s_a_empty[h][s]), 1);
      }
    for (int s = 0; s < kWeightSlots; ++s) {
      mbar_init(smem_u32(&s_w_full[s]), 1);
      mbar_init(smem_u32(&s_w_empty[s]), halves);
    }
    for (int b = 0; b < 2; ++b) {
      for (int h = 0; h < 2; ++h) {
        mbar_init(smem_u32(&s_acc_full[b][h]), 1);
        mbar_init(smem_u32(&s_acc_empty[b][h]), 4);
      }
      mbar_init(smem_u32(&s_part[b]), 4 * halves);
      mbar_init(smem_u32(&s_place_full[b]), 4 * halves);
      // read by the gather warps, the MMA issuers and the weight warp; the run warp has read it when the gather has its runs
      mbar_init(smem_u32(&s_place_empty[b]), 4 * kTeams * halves + halves + (STREAM ? 1 : 0));
    }
    mbar_init_fence();
  }
  if (warp == kMmaWarp) {
    tmem_alloc(smem_u32(&s_tmem_base), 512u);
    tmem_relinquish();
  }
  after_previous<false>();                     // nothing before this reads what another kernel writes
  if (tid < 64) {
    s_epi[tid] = (tid < p.N && p.scale) ? __ldg(p.scale + tid) : 1.f;
    s_epi[64 + tid] = tid < p.N ? p.bias.at<!I8>(tid) : 0.f;
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = uniform(s_tmem_base);
  const uint32_t tmem_a = tmem_base + 256u;          // operands behind the 2 buffers x 2 halves x 64 accumulator columns
  volatile int* abort_flag = &s_abort;
  const int tile_rows = halves * kHalfRows;
  const int my_tiles = (p.num_tiles - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;
  const uint32_t place_full0 = smem_u32(s_place_full), place_empty0 = smem_u32(s_place_empty);
  auto tile_row = [&](int ti) { return ((int64_t)blockIdx.x + (int64_t)ti * gridDim.x) * tile_rows; };

  if (warp < kMmaWarp) {
    // ======================= gather =======================
    const int h = warp >> 2 & 1, rows_of = warp & 7, team = warp >> 3;
    if (h < halves) {
      const uint32_t a_lane = tmem_a + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)(h * kOperands * kOperandCols);
      const uint32_t a_full0 = smem_u32(&s_a_full[h][0]), a_empty0 = smem_u32(&s_a_empty[h][0]);
      const uint32_t run_full0 = smem_u32(s_run_full), run_empty0 = smem_u32(s_run_empty);
      const uint32_t run0 = base_u + (uint32_t)p.run_off;
      const bool one = elect_one();
      int slot = 0;
      uint32_t run_par = 0u;
      uint32_t count = 0u;                            // batches of this half so far; batch c is operand c % kOperands
      uint32_t sent = 0u;                             // operand that is written but not reported, plus one
      bool dead = false;
#ifdef SPH_TEST_HOOKS
      int withhold = p.test_withhold ? 2 : 0;         // test build only: the second operand is never reported
#endif
      auto report = [&]() {
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        const uint32_t at = sent - 1u;
        sent = 0u;
#ifdef SPH_TEST_HOOKS
        if (withhold > 0 && --withhold == 0 && warp == 0) return;
#endif
        if (one) mbar_arrive(a_full0 + 8u * at);
      };
#pragma unroll 1
      for (int ti = 0; ti < my_tiles && !dead; ++ti) {
        const int pb = ti & 1;
        if (!warp_wait(place_full0 + 8u * pb, ((uint32_t)ti >> 1) & 1u, abort_flag)) break;
        const Plan* plan = s_plan + pb;
        const uint32_t offsets = uniform(h ? plan->offsets1 : plan->offsets0);
#pragma unroll 1
        for (int l = 0; l < kLines; ++l) {
          const uint32_t lo = uniform(plan->lo[l]);
          const int hi = (int)uniform((uint32_t)plan->hi[l]);
          const bool any = hi >= 0;                   // some row of the tile has an entry in this line
          if (any) {
            if (sent) report();
            if (!warp_wait(run_full0 + 8u * slot, run_par, abort_flag)) { dead = true; break; }
          }
          const bool split = any && (uint32_t)hi - lo >= cap;
          const uint32_t run = run0 + (uint32_t)slot * slot_bytes;
          const uint32_t line_offsets = (offsets >> (l * L)) & ((1u << L) - 1u);
          const int n = __popc(line_offsets);
          int j = (int)((count ^ (uint32_t)team) & 1u) * U;            // first place of this team's next batch
          uint32_t c = count + (uint32_t)(j / U);
          count += (uint32_t)((n + U - 1) / U);
          uint32_t next[U];                           // a batch ahead, what says where its rows are
          auto hand_over = [&](const uint4 (&v)[8]) {
            if (sent) report();                       // behind this batch's loads
            const uint32_t op = c % kOperands;
            if (!warp_wait(a_empty0 + 8u * op, (c / kOperands & 1u) ^ 1u, abort_flag)) return false;
            tc_fence_after();
            tmem_st_batch(a_lane + op * kOperandCols, v);
            sent = op + 1u;
            j += kTeams * U;
            c += kTeams;
            return true;
          };
          if (!split) {                               // their places
            const uint16_t* place = s_place + ((pb * 8 + rows_of) * kLines + l) * (LP * 32) + lane;
#pragma unroll
            for (int u = 0; u < U; ++u) next[u] = place[(j + u) * 32];        // behind the line: something unused
#pragma unroll 1
            while (j < n) {
              uint4 v[8];                             // U rows of KC pieces
#pragma unroll
              for (int u = 0; u < U; ++u) {
                const uint32_t at = run + next[u] * 16u;
#pragma unroll
                for (int q = 0; q < KC; ++q) v[u * KC + q] = lds128(at ^ (uint32_t)(q << 4), next[u] != kAbsent);
              }
#pragma unroll
              for (int u = 0; u < U; ++u) next[u] = place[(j + kTeams * U + u) * 32];
              if (!hand_over(v)) { dead = true; break; }
            }
          } else {                                    // the buffer does not hold the run: the table's entries
            const uint32_t held = held_of_split(lo, hi, cap);          // rows from lo on that it holds
            const bool whole = ((uintptr_t)p.rows & 31u) == 0;
            const int64_t r = tile_row(ti) + rows_of * 32 + lane;
            uint32_t todo = line_offsets;
            auto drop = [&]() {                       // the other team's batch
#pragma unroll
              for (int u = 0; u < U; ++u) todo &= todo - 1u;
            };
            auto entries = [&]() {
#pragma unroll
              for (int u = 0; u < U; ++u) {
                const int k = l * L + __ffs((int)todo) - 1;
                const bool some = todo != 0u && r < p.n_out;
                next[u] = some ? (uint32_t)__ldg(p.nbr + (int64_t)(p.flip_k ? KV - 1 - k : k) * p.n_out + r) : ~0u;
                if (next[u] >= (uint32_t)p.n_rows) next[u] = ~0u;
                todo &= todo - 1u;
              }
              drop();
            };
            if (j) drop();
            entries();
#pragma unroll 1
            while (j < n) {
              uint4 v[8];
#pragma unroll
              for (int u = 0; u < U; ++u) {
                const uint32_t i = next[u] - lo, at = run + row_at<KC>(i);
#pragma unroll
                for (int q = 0; q < KC; ++q) v[u * KC + q] = lds128(at ^ (uint32_t)(q << 4), i < held);
              }
#pragma unroll
              for (int u = 0; u < U; ++u) {
                const bool beyond = next[u] != ~0u && next[u] - lo >= held;
                const uint8_t* src = (const uint8_t*)p.rows + (size_t)next[u] * ROW;
#pragma unroll
                for (int q = 0; q < KC; q += 2) ldg256(v[u * KC + q], v[u * KC + q + 1], src + q * 16, beyond, whole);
              }
              entries();
              if (!hand_over(v)) { dead = true; break; }
            }
          }
          if (dead) break;
          if (any) {
            __syncwarp();
            if (one) mbar_arrive(run_empty0 + 8u * slot);
            if (++slot == p.run_slots) { slot = 0; run_par ^= 1u; }
          }
        }
        if (dead) break;
        if (sent) report();
        if (one) mbar_arrive(place_empty0 + 8u * pb);
      }
    }
  } else if (warp < kEpiWarp) {
    // ======================= MMA issuers: one warp per half =======================
    const int h = warp - kMmaWarp;
    if (h < halves) {
      const bool one = elect_one();
      const uint32_t idesc = I8 ? make_idesc(2u, 1u, 0u, 0u, kHalfRows, (uint32_t)p.N)
                                : make_idesc(1u, p.is_bf16 ? 1u : 0u, 0u, 0u, kHalfRows, (uint32_t)p.N);
      const uint32_t lbo_w = (uint32_t)(p.N / 8) * 128u;
      const uint64_t w_desc0 = make_smem_desc(base_u + (uint32_t)p.w_off, lbo_w, 128u);
      const uint64_t w_hi = w_desc0 & 0xffffffff00000000ull;
      const uint32_t w_lo0 = (uint32_t)w_desc0;
      const uint32_t w_step = (2u * lbo_w) >> 4;                 // 32 bytes of K per instruction
      const uint32_t w_units = (uint32_t)p.w_bytes >> 4;
      const uint32_t a_full0 = smem_u32(&s_a_full[h][0]), a_empty0 = smem_u32(&s_a_empty[h][0]);
      const uint32_t w_full0 = smem_u32(s_w_full), w_empty0 = smem_u32(s_w_empty);
      const uint32_t a0 = tmem_a + (uint32_t)(h * kOperands * kOperandCols);
      int ws = 0;
      uint32_t w_par = 0u, count = 0u;               // count: batches of this half so far
      bool dead = false, seen = false;                // seen: the next offset's barriers are complete
      if (!STREAM) dead = !warp_wait(w_full0, 0u, abort_flag);
      for (int ti = 0; ti < my_tiles && !dead; ++ti) {
        const int buf = ti & 1;
        if (!warp_wait(place_full0 + 8u * buf, ((uint32_t)ti >> 1) & 1u, abort_flag)) break;
        const uint32_t o0 = uniform(s_plan[buf].offsets0), o1 = uniform(s_plan[buf].offsets1);
        if (one) mbar_arrive(place_empty0 + 8u * buf);
        const uint32_t own = h ? o1 : o0;
        const uint32_t walk = STREAM && halves == 2 ? o0 | o1 : own;        // streamed images come for both halves
        if (!warp_wait(smem_u32(&s_acc_empty[buf][h]), (((uint32_t)ti >> 1) & 1u) ^ 1u, abort_flag)) break;
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + (uint32_t)((buf * 2 + h) * 64);
        uint32_t acc = 0u;
        if constexpr (STREAM) {
          uint32_t todo = walk;
          int k = __ffs((int)todo) - 1;
#pragma unroll 1
          while (todo) {
            const uint32_t op = count % kOperands;
            const bool mine = own >> k & 1u;
            if (!__all_sync(0xffffffffu, seen)) {
              if (!warp_wait(w_full0 + 8u * ws, w_par, abort_flag)) { dead = true; break; }
              if (mine && !warp_wait(a_full0 + 8u * op, count / kOperands & 1u, abort_flag)) { dead = true; break; }
            }
            tc_fence_after();
            if (one) {
              if (mine) {
                const uint32_t w_lo = w_lo0 + (uint32_t)ws * w_units;
#pragma unroll
                for (int j = 0; j < KC / 2; ++j)
                  umma_ta<I8>(d_tmem, a0 + op * kOperandCols + (uint32_t)(j * 8), w_hi | (uint64_t)(w_lo + (uint32_t)j * w_step), idesc,
                              j ? 1u : acc);
                umma_commit(a_empty0 + 8u * op);
                umma_commit(w_empty0 + 8u * ws);
              } else {
                mbar_arrive(w_empty0 + 8u * ws);
              }
            }
            if (mine) {
              acc = 1u;
              ++count;
            }
            if (++ws == p.weight_slots) { ws = 0; w_par ^= 1u; }
            todo &= todo - 1u;
            k = __ffs((int)todo) - 1;
            // looked at now, the barriers of the next offset are known to be complete without the 90 cycles a wait takes for each
            seen = mbar_test_wait(a_full0 + 8u * (count % kOperands), count / kOperands & 1u) &
                   mbar_test_wait(w_full0 + 8u * ws, w_par);
          }
        } else {
#pragma unroll 1
          for (int l = 0; l < kLines && !dead; ++l) {
            uint32_t todo = (own >> (l * L)) & ((1u << L) - 1u);
#pragma unroll 1
            while (todo) {
              int k[U];                               // offsets of the batch in the line, -1: no more
#pragma unroll
              for (int u = 0; u < U; ++u) {
                k[u] = todo ? __ffs((int)todo) - 1 : -1;
                todo &= todo - 1u;
              }
              const uint32_t op = count % kOperands;
              if (!warp_wait(a_full0 + 8u * op, count / kOperands & 1u, abort_flag)) { dead = true; break; }
              tc_fence_after();
              if (one) {
#pragma unroll
                for (int u = 0; u < U; ++u) {
                  if (u == 0 || k[u] >= 0) {
                    const uint32_t w_lo = w_lo0 + (uint32_t)(l * L + k[u]) * w_units;
#pragma unroll
                    for (int j = 0; j < KC / 2; ++j)
                      umma_ta<I8>(d_tmem, a0 + op * kOperandCols + (uint32_t)(u * KC * 4 + j * 8),
                                  w_hi | (uint64_t)(w_lo + (uint32_t)j * w_step), idesc, u || j ? 1u : acc);
                  }
                }
                umma_commit(a_empty0 + 8u * op);
              }
              acc = 1u;
              ++count;
            }
          }
        }
        if (!dead && one) umma_commit(smem_u32(&s_acc_full[buf][h]));
      }
    }
  } else if (warp < kRunWarp) {
    // ======================= epilogue =======================
    const int q = warp & 3;                       // TMEM lane quarter this warp may read: rows 32q .. 32q+31 of a half
    // Rows of 80 to 128 bytes go through shared memory, an odd number of 16-byte pieces apart: stored by the lane that has them, a
    // store instruction touches 32 lines and takes 37 turns of the data path that the gather waits for, staged 12 (64 -> 64
    // channels of fp16: 177 -> 162 us).  Narrower rows do not repay the instructions (32 -> 32: 205 against 208).
    const int pieces = p.N * p.out_esize / 16, pitch = pieces | 1;
    const bool staged = p.stage_off >= 0;
    uint4* stage = (uint4*)(base + (staged ? p.stage_off : 0)) + q * 32 * (kStagePieces + 1);
    const bool one = elect_one();
    bool dead = false;
    for (int ti = 0; ti < my_tiles && !dead; ++ti) {
      const int buf = ti & 1;
#pragma unroll 1
      for (int h = 0; h < halves; ++h) {
        if (!warp_wait(smem_u32(&s_acc_full[buf][h]), ((uint32_t)ti >> 1) & 1u, abort_flag)) { dead = true; break; }
        tc_fence_after();
        const int64_t row0 = tile_row(ti) + h * kHalfRows + q * 32;
        const uint32_t taddr = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)((buf * 2 + h) * 64);
        const int rows = row0 < p.n_out ? (int)min((int64_t)32, p.n_out - row0) : 0;
        uint4* dst = (uint4*)((uint8_t*)p.out + row0 * p.N * p.out_esize);
#pragma unroll 1
        for (int c0 = 0, c = 0; c0 < p.N && rows > 0; c0 += 16) {
          uint32_t raw[16];
          tmem_ld16(taddr + (uint32_t)c0, raw);     // this thread's row, channels c0 .. c0+15
          tmem_ld_wait();
          uint4 piece[4];
          const int n = convert16<I8>(piece, p.out_dtype, raw, s_epi + c0, s_epi + 64 + c0, p.relu);
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            if (j >= n) break;
            if (staged) stage[lane * pitch + c + j] = piece[j];
            else if (lane < rows) dst[lane * pieces + c + j] = piece[j];
          }
          c += n;
        }
        if (staged) {                               // the rows are consecutive: 512 bytes a store
          __syncwarp();
          const int n = rows * pieces;
          for (int i = lane; i < n; i += 32) dst[i] = stage[i / pieces * pitch + i % pieces];
          __syncwarp();
        }
        tc_fence_before();
        __syncwarp();
        if (one) mbar_arrive(smem_u32(&s_acc_empty[buf][h]));
      }
    }
  } else if (warp == kRunWarp) {
    // ======================= runs of input rows =======================
    const bool one = elect_one();
    int slot = 0;
    uint32_t par = 1u;
    bool dead = false;
    for (int ti = 0; ti < my_tiles && !dead; ++ti) {
      if (!warp_wait(place_full0 + 8u * (ti & 1), ((uint32_t)ti >> 1) & 1u, abort_flag)) break;
      const Plan plan = s_plan[ti & 1];
#pragma unroll
      for (int l = 0; l < kLines; ++l) {
        const int hi = (int)uniform((uint32_t)plan.hi[l]);
        const uint32_t lo = uniform(plan.lo[l]);
        if (hi < 0 || dead) continue;
        if (!warp_wait(smem_u32(&s_run_empty[0]) + 8u * slot, par, abort_flag)) { dead = true; continue; }
        if (one) {
          const uint32_t span = (uint32_t)hi - lo + 1u;
          const uint32_t len = span <= cap ? span : held_of_split(lo, hi, cap);
          const uint32_t boxes = (len + kBox - 1) / kBox;
          const uint32_t full = smem_u32(&s_run_full[0]) + 8u * slot;
          uint32_t dst = base_u + (uint32_t)p.run_off + (uint32_t)slot * slot_bytes;
          if (boxes == 0) mbar_arrive(full);
          else mbar_arrive_expect_tx(full, boxes * (kBox * ROW));
          for (uint32_t b = 0; b < boxes; ++b, dst += kBox * ROW) tma_rows(dst, &map, (int)(lo + b * kBox), full);
        }
        __syncwarp();
        if (++slot == p.run_slots) { slot = 0; par ^= 1u; }
      }
    }
  } else if (warp == kWeightWarp) {
    // ======================= weight images =======================
    const uint32_t w_full0 = smem_u32(s_w_full), w_empty0 = smem_u32(s_w_empty);
    const uint32_t w_smem = base_u + (uint32_t)p.w_off;
    const bool one = elect_one();
    if (!STREAM) {
      if (one) {
        mbar_arrive_expect_tx(w_full0, (uint32_t)(KV * p.w_bytes));
        for (int k = 0; k < KV; ++k)
          bulk_g2s(w_smem + (uint32_t)(k * p.w_bytes), (const uint8_t*)p.packed + (size_t)k * p.w_bytes, (uint32_t)p.w_bytes, w_full0);
      }
    } else {
      int ws = 0;
      uint32_t par = 1u;
      bool dead = false;
      for (int ti = 0; ti < my_tiles && !dead; ++ti) {
        if (!warp_wait(place_full0 + 8u * (ti & 1), ((uint32_t)ti >> 1) & 1u, abort_flag)) break;
        const uint32_t o0 = uniform(s_plan[ti & 1].offsets0), o1 = uniform(s_plan[ti & 1].offsets1);
        if (one) mbar_arrive(place_empty0 + 8u * (ti & 1));
        uint32_t walk = halves == 2 ? o0 | o1 : o0;
#pragma unroll 1
        while (walk) {
          const int k = __ffs((int)walk) - 1;
          walk &= walk - 1u;
          if (!warp_wait(w_empty0 + 8u * ws, par, abort_flag)) { dead = true; break; }
          if (one) {
            mbar_arrive_expect_tx(w_full0 + 8u * ws, (uint32_t)p.w_bytes);
            bulk_g2s(w_smem + (uint32_t)(ws * p.w_bytes), (const uint8_t*)p.packed + (size_t)k * p.w_bytes, (uint32_t)p.w_bytes,
                     w_full0 + 8u * ws);
          }
          __syncwarp();
          if (++ws == p.weight_slots) { ws = 0; par ^= 1u; }
        }
      }
    }
  } else {
    // ======================= planning =======================
    const int w = warp - kPlanWarp;               // rows of gather warp w
    if (w < 4 * halves) {
      const uint32_t n_rows_u = (uint32_t)p.n_rows;
      const uint32_t part0 = smem_u32(s_part);
      const bool one = elect_one();
      uint32_t bad = 0u;
      int entry[KV];
      auto load = [&](int ti) {
        const int64_t r = tile_row(ti) + w * 32 + lane;
        const bool ok = ti < my_tiles && r < p.n_out;
        const int64_t step = p.flip_k ? -p.n_out : p.n_out;
        const int* at = p.nbr + (p.flip_k ? (int64_t)(KV - 1) * p.n_out : 0) + r;
#pragma unroll
        for (int k = 0; k < KV; ++k) {
          entry[k] = ok ? __ldg(at) : -1;
          at += step;
        }
      };
      // The lines of memory that hold a tile's entries, to L2: lane k those of offset k.
      auto prefetch = [&](int ti) {
        const int64_t r = tile_row(ti) + w * 32;
        if (ti < my_tiles && r < p.n_out && lane < KV) {
          const int* at = p.nbr + (int64_t)lane * p.n_out + r;
          asm volatile("prefetch.global.L2 [%0];" ::"l"(at));
          if (r + 32 <= p.n_out) asm volatile("prefetch.global.L2 [%0];" ::"l"(at + 31));
        }
      };
      load(0);
      prefetch(1);
#pragma unroll 1
      for (int ti = 0; ti < my_tiles; ++ti) {
        const int pb = ti & 1;
        Partial* part = s_partial + pb * 8;
        prefetch(ti + 2);
        uint32_t absent = 0u;                         // bit KV - 1 - k: no neighbour at offset k
        int least = 0, most = -1;
#pragma unroll
        for (int k = 0; k < KV; ++k) {
          least = min(least, entry[k]);
          most = max(most, entry[k]);
        }
        if (__any_sync(0xffffffffu, least < -1 || most >= (int)n_rows_u)) {      // ids that are no rows count as absent
          bad = 1u;
#pragma unroll
          for (int k = 0; k < KV; ++k)
            if ((uint32_t)entry[k] >= n_rows_u) entry[k] = -1;
        }
#pragma unroll
        for (int l = 0; l < kLines; ++l) {
          uint32_t lo = ~0u;
          int hi = -1;
#pragma unroll
          for (int o = 0; o < L; ++o) {
            const int v = entry[l * L + o];
            lo = min(lo, (uint32_t)v);
            hi = max(hi, v);
            absent = __funnelshift_l((uint32_t)v, absent, 1);
          }
          lo = __reduce_min_sync(0xffffffffu, lo);
          hi = __reduce_max_sync(0xffffffffu, hi);
          if (one) part[w].run[l] = make_int2((int)lo, hi);
        }
        const uint32_t present = __brev(__reduce_or_sync(0xffffffffu, ~absent & ((1u << KV) - 1u))) >> (32 - KV);
        if (one) {
          part[w].offsets = present;
          mbar_arrive(part0 + 8u * pb);
        }
        __syncwarp();
        if (!warp_wait(part0 + 8u * pb, ((uint32_t)ti >> 1) & 1u, abort_flag)) break;
        const Plan plan = combine(part, lane);
        // everyone is done with the plan of the tile before last
        if (!warp_wait(place_empty0 + 8u * pb, (((uint32_t)ti >> 1) & 1u) ^ 1u, abort_flag)) break;
        if (w == 0 && one) s_plan[pb] = plan;
        const uint32_t offsets = w < 4 ? plan.offsets0 : plan.offsets1;
#pragma unroll
        for (int l = 0; l < kLines; ++l) {
          uint16_t* place = s_place + ((pb * 8 + w) * kLines + l) * (LP * 32) + lane;
          // the gather reads the table itself for a run that the buffer does not hold
          if (plan.hi[l] >= 0 && (uint32_t)plan.hi[l] - plan.lo[l] >= cap) continue;
#pragma unroll
          for (int o = 0; o < L; ++o) {
            if (offsets >> (l * L + o) & 1u) {
              const int v = entry[l * L + o];
              *place = (uint16_t)(v < 0 ? kAbsent : row_at<KC>((uint32_t)v - plan.lo[l]) >> 4);
              place += 32;
            }
          }
          if (U > 1) {                                // the rest of the last batch
            const int n = __popc(offsets >> (l * L) & ((1u << L) - 1u));
            for (int u = n; u % U != 0; ++u, place += 32) *place = (uint16_t)kAbsent;
          }
        }
        __syncwarp();
        if (one) mbar_arrive(place_full0 + 8u * pb);
        load(ti + 1);
      }
      if (bad && one && p.status) atomicOr(p.status, SPH_STATUS_BAD_INDEX);
    }
  }

  // ---- wind down: every thread arrives here, also after an abort
  tc_fence_before();
  __syncthreads();
  if (s_abort) {
    // let copies still in flight land before the CTA's shared memory is released
    const long long t0 = clock64();
    while (clock64() - t0 < 4000000ll) { }
    if (tid == 0 && p.status) atomicOr(p.status, SPH_STATUS_TIMEOUT);
    __syncthreads();
  }
  if (warp == kMmaWarp) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512u);
  }
}

// Dynamic shared memory, from the aligned base: plans, epilogue constants, places, weights, runs.
bool plan_smem(TmemParams* p, int kv, int row_bytes, int* smem_bytes) {
  const int batch = 128 / row_bytes, line = div_up(kv / kLines, batch) * batch;
  int off = 0;
  p->plan_off = off; off += 2 * (int)sizeof(Plan);
  p->part_off = off; off += 2 * 8 * (int)sizeof(Partial);
  p->epi_off = off; off += 2 * 64 * (int)sizeof(float);
  const int pieces = p->N * p->out_esize / 16;
  p->stage_off = -1;
  if (pieces > kStagePieces / 2 && pieces <= kStagePieces) {
    p->stage_off = off;
    off += 4 * 32 * (kStagePieces + 1) * 16;
  }
  p->place_off = off; off += 2 * 8 * kLines * line * 32 * (int)sizeof(uint16_t);
  off = (off + 127) & ~127;
  p->w_off = off;
  // Where there are more input rows than output rows the runs are longer: room for them rather than for weights or a third run.
  // 128-byte rows, four images instead of eight (448 -> 576 rows at 64 channels of fp16): input gradients of strides (1,1,4) and (1,1,2)
  // 83 -> 70 and 106 -> 102 us; but 64 -> 64 on 683 k rows whose runs fit 166 -> 173.  Two runs of 512 rows instead of three of
  // 352 (32 -> 64): strided, 683 k rows, 131 -> 122 us, surfaces, 146 k rows, 44 -> 40; with fewer input rows than output rows 456 -> 488.
  p->weight_slots = p->n_rows > p->n_out ? kWeightSlots / 2 : kWeightSlots;
  off += (row_bytes == 128 ? p->weight_slots : kv) * p->w_bytes;
  p->run_off = (off + 1023) & ~1023;
  const int bytes = kSmemTotal - 1024 - p->run_off;
  p->run_slots = row_bytes == 128 || (p->n_rows > p->n_out && bytes / (kRunSlots * row_bytes) < 512) ? 2 : kRunSlots;
  const int rows = bytes / (p->run_slots * row_bytes) / kBox * kBox;
  p->cap = rows > 1024 ? 1024 : rows;
  *smem_bytes = 1024 + p->run_off + p->run_slots * p->cap * row_bytes;
  return p->cap >= 256;               // runs of 256 output rows are 260 to 450 rows long
}

bool shape_ok(int dtype, int kv, int K, int N) {
  if (dtype != SPH_F16 && dtype != SPH_BF16 && dtype != SPH_I8) return false;
  const int row_bytes = K * dtype_bytes(dtype);
  return (kv == 27 || kv == 9) && (row_bytes == 32 || row_bytes == 64 || row_bytes == 128) && N % 16 == 0 && N >= 16 && N <= 64;
}

using EncodeTiled = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                 const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                 CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiled encode_tiled() {
  static const EncodeTiled fn = [] {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult found;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &f, 12000, cudaEnableDefault, &found) != cudaSuccess ||
        found != cudaDriverEntryPointSuccess)
      f = nullptr;
    return (EncodeTiled)f;
  }();
  return fn;
}

}  // namespace tmemform
}  // namespace

bool conv_tmem_supported(int dtype, int kv, int K, int N) { return tmemform::shape_ok(dtype, kv, K, N); }

int conv_gather_tmem(const void* rows, int dtype, int64_t n_rows, const void* packed, const int* nbr, int64_t n_out, int kv,
                     int K, int N, int flip_k, const float* scale, Bias bias, int relu, void* out, int out_dtype, int* status,
                     cudaStream_t st) {
  using namespace tmemform;
  if (!shape_ok(dtype, kv, K, N) || n_rows < 1) {
    set_error("conv_gather_tmem: unsupported dtype/shape");
    return SPH_ERR_UNSUPPORTED;
  }
  const int row_bytes = K * dtype_bytes(dtype);
  TmemParams p;
  p.rows = rows; p.packed = packed; p.nbr = nbr;
  p.n_rows = n_rows; p.n_out = n_out;
  p.N = N; p.flip_k = flip_k;
  p.w_bytes = N * row_bytes;
  p.is_bf16 = dtype == SPH_BF16;
  p.scale = scale; p.bias = bias; p.relu = relu;
  p.out = out; p.out_dtype = out_dtype; p.out_esize = dtype_bytes(out_dtype); p.status = status;
#ifdef SPH_TEST_HOOKS
  p.test_withhold = g_test_withhold;
#endif
  int smem_bytes = 0;
  if (!plan_smem(&p, kv, row_bytes, &smem_bytes)) {
    set_error("conv_gather_tmem: operands do not fit in shared memory");
    return SPH_ERR_UNSUPPORTED;
  }
  const int sms = current_sm_count();
  if (sms <= 0) return SPH_ERR_CUDA;
  // Every CTA takes all 512 TMEM columns, so exactly one is resident per SM.  Tiles of one half where those of two would leave
  // half of the SMs idle: 64 -> 64 on 9 k / 19 k / 23 k rows 17.4 / 20.5 / 22.5 us with one, 21.5 / 22.5 / 21.5 with two; 32 -> 32
  // 14.4 / 16.4 / 17.3 and 16.4 / 16.5 / 16.6.
  p.halves = div_up64(n_out, 2 * kHalfRows) > sms / 2 ? 2 : 1;
  p.num_tiles = (int)div_up64(n_out, p.halves * kHalfRows);
  const int grid = sms < p.num_tiles ? sms : p.num_tiles;
  if (grid < 1) return SPH_OK;

  const EncodeTiled encode = encode_tiled();
  if (encode == nullptr) {
    set_error("conv_gather_tmem: the driver has no cuTensorMapEncodeTiled");
    return SPH_ERR_CUDA;
  }
  CUtensorMap map;
  const cuuint64_t dims[2] = {(cuuint64_t)row_bytes, (cuuint64_t)n_rows}, strides[1] = {(cuuint64_t)row_bytes};
  const cuuint32_t box[2] = {(cuuint32_t)row_bytes, kBox}, steps[2] = {1, 1};
  const CUtensorMapSwizzle swizzle = row_bytes == 128  ? CU_TENSOR_MAP_SWIZZLE_128B
                                     : row_bytes == 64 ? CU_TENSOR_MAP_SWIZZLE_64B
                                                       : CU_TENSOR_MAP_SWIZZLE_32B;
  const CUresult rc = encode(&map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(rows), dims, strides, box, steps,
                             CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (rc != CUDA_SUCCESS) {
    set_error("conv_gather_tmem: cuTensorMapEncodeTiled failed (%d)", (int)rc);
    return SPH_ERR_CUDA;
  }
#define SPH_TMEM_LAUNCH(KC_, I8_, L_)                                                                    \
  do {                                                                                                   \
    SPH_CUDA(allow_smem(conv_gather_tmem_kernel<KC_, I8_, L_>, kSmemTotal));                             \
    launch(conv_gather_tmem_kernel<KC_, I8_, L_>, grid, kThreads, smem_bytes, st, map, p);                   \
  } while (0)
#define SPH_TMEM_ROWS(I8_, L_)                        \
  switch (row_bytes) {                                \
    case 32: SPH_TMEM_LAUNCH(2, I8_, L_); break;      \
    case 64: SPH_TMEM_LAUNCH(4, I8_, L_); break;      \
    default: SPH_TMEM_LAUNCH(8, I8_, L_);             \
  }
  if (dtype == SPH_I8) {
    if (kv == 27) { SPH_TMEM_ROWS(true, 9) } else { SPH_TMEM_ROWS(true, 3) }
  } else {
    if (kv == 27) { SPH_TMEM_ROWS(false, 9) } else { SPH_TMEM_ROWS(false, 3) }
  }
#undef SPH_TMEM_ROWS
#undef SPH_TMEM_LAUNCH
  SPH_LAUNCH_CHECK();
  return SPH_OK;
}

}  // namespace sph
