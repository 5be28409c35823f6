// Grouped products of a mixture of experts for prompts, bf16, on the 5th-generation tensor cores: the (token, expert) pairs'
// rows lie expert by expert (moe_align, moe_gather), and for every row r of expert e
//   first product:   hidden[r, f] = join(gate[e, f] . a[r], up[e, f] . a[r])     or   max(up[e, f] . a[r], 0)^2
//   second product:  out[r, n] = down[e, n] . hidden[r]
// in one launch each, the activation formed from the 32-bit sums.
//
// The experts' rows are few and uneven (256 on average where 2,048 tokens choose 4 of 32 experts), so they are the tensor
// pipe's N, which may be any multiple of 16 up to 256, and the weights its M: a block multiplies two tiles of 128 weight
// rows (a gate tile and the up tile beside it, or two neighbouring ones) with up to NT rows of one expert.  An expert's
// rows are cut into equal tiles (moe_align's table), nothing is multiplied that is not there but a run's last few rows up to
// 16, and the host need not know the experts' loads.
//
// One block an SM; the blocks take (expert, weight tile, row tile) in turn, the row tiles of a weight tile next to one another
// so that weights come from memory once.  Warp 0 brings both weight tiles and the rows by TMA, 64 k a stage; warp 1 issues the
// products (two accumulators of NT columns in tensor memory); warps 4 to 11 take the accumulators out, join and store them
// (a lane owns a weight row, so a warp stores 64 neighbouring bytes of a row).  The ring runs on from item to item; with up to
// 128 rows two pairs of accumulators alternate.
//
// What bounds it: with many rows the shared memory, which takes 48 to 64 KB a stage in and gives every weight tile and all rows
// to the products four times; with few the passes over the weights.  32 experts of 3,584 at width 4,096, 4 a token, whole
// call with the choices given (B200, call after call): 2,048 tokens 763 us where two batched library products at a common
// stride and an activation between them took 878 (the products 444 and 225 us for 494, 38 and 231); 1,000 tokens 550 and
// 648; 130 tokens 458 and 532 (430 of bytes).  16 warps that take the accumulators out: the same.
#include <cuda.h>
#include <string.h>

#include "common.cuh"
#include "sm100.cuh"

#define MG_K 64
#define MG_W_BYTES (128 * MG_K * 2)         // one weight tile of a stage
#define MG_OUT_WARPS 8
#define MG_THREADS (128 + 32 * MG_OUT_WARPS)
#define MG_SPIN_LIMIT (1u << 20)

#define MG_SILU 0
#define MG_CLAMPED 1
#define MG_SQUARED 2
#define MG_PLAIN 3

struct GroupedParams {
  bf16* out;                                // [rows, width]
  const int4* tiles;                        // {expert, first row, rows | row tiles of the expert << 12, the expert's first tile}
  const int* meta;                          // [1]: how many
  int width;                                // outputs of an expert
  int weight_rows, second;                  // rows of an expert's matrix; the second tile's distance from the first
  int weight_tiles, k_stages;
  float alpha, limit, shift;
  int* status;
};

template <int NT> struct GroupedRing {
  static constexpr int STAGE = 2 * MG_W_BYTES + NT * MG_K * 2;
  static constexpr int STAGES = NT >= 256 ? 3 : NT >= 128 ? 4 : 5;
  static constexpr int BUFFERS = NT >= 256 ? 1 : 2;          // pairs of accumulators
  static constexpr int BYTES = STAGES * STAGE + 256;
};

__device__ __forceinline__ void mg_ld16(unsigned taddr, float (&v)[16]) {
  unsigned* r = reinterpret_cast<unsigned*>(v);
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                 "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]) : "r"(taddr));
}

template <int NT, int MODE>
__global__ void __launch_bounds__(MG_THREADS, 1)
moe_grouped_kernel(const __grid_constant__ CUtensorMap w_map, const __grid_constant__ CUtensorMap a_map, const GroupedParams p) {
  using Ring = GroupedRing<NT>;
  constexpr int STAGES = Ring::STAGES, BUFFERS = Ring::BUFFERS;
  constexpr bool JOINED = MODE == MG_SILU || MODE == MG_CLAMPED;
  constexpr int COVERS = JOINED ? 128 : 256;                 // outputs of an item
  KVB_KERNEL_PROLOGUE(KVB_TAG_MOE_GEMM);
  extern __shared__ __align__(1024) unsigned char mg_dyn[];
  unsigned long long* full = reinterpret_cast<unsigned long long*>(mg_dyn + STAGES * Ring::STAGE);
  unsigned long long* empty = full + STAGES;
  unsigned long long* acc_full = empty + STAGES;             // [BUFFERS]
  unsigned long long* acc_empty = acc_full + BUFFERS;        // [BUFFERS] the warps that take them out
  unsigned long long* drain = acc_empty + BUFFERS;           // given up: products in flight
  unsigned* tmem_slot = reinterpret_cast<unsigned*>(drain + 1);
  int* abort_flag = reinterpret_cast<int*>(tmem_slot + 1);
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  if (kvb_smem(mg_dyn) & 1023u) {                            // cannot happen with the alignment asked for; never run misaligned
    if (threadIdx.x == 0) atomicOr(p.status, KVB_STATUS_WAIT_TIMEOUT);
    return;
  }
  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) { kvb_mbar_init(&full[s], 1); kvb_mbar_init(&empty[s], 1); }
    for (int b = 0; b < BUFFERS; ++b) { kvb_mbar_init(&acc_full[b], 1); kvb_mbar_init(&acc_empty[b], MG_OUT_WARPS); }
    kvb_mbar_init(drain, 1);
    *abort_flag = 0;
    kvb_mbar_init_fence();
  }
  if (warp == 1) kvb_tc5_alloc(tmem_slot, 512u);
  kvb_tc5_fence_before();
  __syncthreads();
  kvb_tc5_fence_after();
  const unsigned tmem = __shfl_sync(0xffffffffu, *tmem_slot, 0);
  auto gave_up = [&] {
    atomicOr(p.status, KVB_STATUS_WAIT_TIMEOUT);
    atomicExch(abort_flag, 1);
  };
  auto aborted = [&] { return *reinterpret_cast<volatile int*>(abort_flag) != 0; };

  const int items = p.meta[1] * p.weight_tiles;
  struct Item { int expert, row0, rows, tile; bool both; };
  auto item = [&](int i) {
    Item it;
    const int4 any = p.tiles[i / p.weight_tiles];            // a row tile of the item's expert
    const int count = any.z >> 12, r = i - any.w * p.weight_tiles;
    it.tile = r / count;
    const int4 mine = p.tiles[any.w + r - it.tile * count];
    it.expert = mine.x;
    it.row0 = mine.y;
    it.rows = mine.z & 0xfff;
    it.both = JOINED || it.tile * COVERS + 128 < p.width;    // the second tile of the last two may lie beyond the matrix
    return it;
  };

  if (warp == 0) {
    // ================= weights and rows =================
    if (lane == 0) {
      int at = 0;                                            // stages asked for so far
      bool ok = true;
      for (int i = blockIdx.x; i < items && ok; i += gridDim.x) {
        const Item it = item(i);
        const int wrow = it.expert * p.weight_rows + it.tile * COVERS, boxes = (it.rows + 63) / 64;
        const unsigned bytes = (it.both ? 2u : 1u) * MG_W_BYTES + boxes * 64 * MG_K * 2;
        for (int k = 0; k < p.k_stages; ++k, ++at) {
          const int s = at % STAGES;
          if (at >= STAGES && !kvb_mbar_wait<MG_SPIN_LIMIT, 4096>(&empty[s], ((at / STAGES) - 1) & 1)) { gave_up(); ok = false; break; }
          if (aborted()) { ok = false; break; }
          unsigned char* to = mg_dyn + s * Ring::STAGE;
          kvb_mbar_expect_tx(&full[s], bytes);
          kvb_tma_2d(to, &w_map, k * MG_K, wrow, &full[s]);
          if (it.both) kvb_tma_2d(to + MG_W_BYTES, &w_map, k * MG_K, wrow + p.second, &full[s]);
          for (int b = 0; b < boxes; ++b)
            kvb_tma_2d(to + 2 * MG_W_BYTES + b * 64 * MG_K * 2, &a_map, k * MG_K, it.row0 + 64 * b, &full[s]);
        }
      }
      if (aborted())                                         // let the copies in flight land before the block may exit
        for (int j = max(0, at - STAGES); j < at; ++j) kvb_mbar_wait<MG_SPIN_LIMIT, 4096>(&full[j % STAGES], (j / STAGES) & 1);
    }
  } else if (warp == 1) {
    // ================= products: the whole warp, one lane issues =================
    const unsigned leader = kvb_elect();
    const unsigned long long base = kvb_tc5_desc(kvb_smem(mg_dyn), 16, 1024);
    unsigned at = 0, n = 0;
    bool ok = true;
    for (int i = blockIdx.x; i < items && ok; i += gridDim.x, ++n) {
      const Item it = item(i);
      const int rows = __shfl_sync(0xffffffffu, it.rows, 0), both = __shfl_sync(0xffffffffu, (int)it.both, 0);
      const unsigned idesc = kvb_tc5_idesc(128, rows, false);
      const unsigned b = n % BUFFERS, acc = tmem + b * 2 * NT;
      if (n >= BUFFERS) ok = __all_sync(0xffffffffu, kvb_mbar_wait<MG_SPIN_LIMIT, 4096>(&acc_empty[b], ((n / BUFFERS) - 1) & 1));
      for (int k = 0; k < p.k_stages && ok; ++k, ++at) {
        const unsigned s = at % STAGES;
        ok = __all_sync(0xffffffffu, kvb_mbar_wait<MG_SPIN_LIMIT, 4096>(&full[s], (at / STAGES) & 1));
        if (!ok) break;
        kvb_tc5_fence_after();
        const unsigned long long w = base + s * (Ring::STAGE / 16), a = w + 2 * MG_W_BYTES / 16;
#pragma unroll
        for (int j = 0; j < 4; ++j) {                        // 16 k: 32 bytes of a row of 128
          kvb_tc5_mma_by(acc, w + 2 * j, a + 2 * j, idesc, k > 0 || j > 0 ? 1u : 0u, leader);
          if (both) kvb_tc5_mma_by(acc + NT, w + MG_W_BYTES / 16 + 2 * j, a + 2 * j, idesc, k > 0 || j > 0 ? 1u : 0u, leader);
        }
        kvb_tc5_commit_by(&empty[s], leader);
      }
      if (ok) kvb_tc5_commit_by(&acc_full[b], leader);
    }
    if (!ok) {
      if (lane == 0) gave_up();
      kvb_tc5_commit_by(drain, leader);                      // tensor memory is given back below: products in flight first
      kvb_mbar_wait<MG_SPIN_LIMIT, 4096>(drain, 0);
    }
    __syncwarp();
  } else if (warp >= 4) {
    // ================= results: 16 rows at a time, turn about between the two warps of a lane quarter =================
    const int quarter = warp & 3, turn = (warp - 4) >> 2;
    const unsigned lanes = (unsigned)(quarter * 32) << 16;
    unsigned n = 0;
    bool ok = true;
    for (int i = blockIdx.x; i < items; i += gridDim.x, ++n) {
      const Item it = item(i);
      const unsigned b = n % BUFFERS;
      ok = __all_sync(0xffffffffu, kvb_mbar_wait<MG_SPIN_LIMIT, 4096>(&acc_full[b], (n / BUFFERS) & 1));
      if (!ok) break;
      kvb_tc5_fence_after();
      const unsigned acc = tmem + lanes + b * 2 * NT;
      const int feature = it.tile * COVERS + quarter * 32 + lane;
      bf16* const to = p.out + (long long)it.row0 * p.width + feature;
      for (int c = turn * 16; c < it.rows; c += 4 * MG_OUT_WARPS) {
        float u[16], v[16];
        mg_ld16(acc + c, u);
        if (it.both) mg_ld16(acc + NT + c, v);
        kvb_tc5_wait_ld();
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          bf16* const at = to + (long long)(c + j) * p.width;
          if (JOINED) {
            float r;
            if (MODE == MG_SILU) {
              r = kvb_silu_for_bf16(u[j]) * v[j];
            } else {
              const float g = fminf(u[j], p.limit);
              r = __fdividef(g, 1.0f + __expf(-p.alpha * g)) * (fminf(fmaxf(v[j], -p.limit), p.limit) + p.shift);
            }
            if (feature < p.width) *at = __float2bfloat16_rn(r);
          } else {
            if (MODE == MG_SQUARED) {
              const float r = fmaxf(u[j], 0.0f), q = fmaxf(v[j], 0.0f);
              u[j] = r * r;
              v[j] = q * q;
            }
            if (feature < p.width) *at = __float2bfloat16_rn(u[j]);
            if (feature + 128 < p.width) at[128] = __float2bfloat16_rn(v[j]);
          }
        }
      }
      kvb_tc5_fence_before();
      __syncwarp();
      if (lane == 0) kvb_mbar_arrive(&acc_empty[b]);
    }
    if (!ok && lane == 0) gave_up();
  }
  kvb_tc5_fence_before();
  __syncthreads();
  if (warp == 1) {
    kvb_tc5_fence_after();
    kvb_tc5_dealloc(tmem, 512u);
  }
}

// Rows of a tile for a batch: `pairs` of `experts`.  Also what moe_align cuts runs by.  Smaller tiles leave room for more stages,
// which keep more of the weights in flight where the rows are few.
extern "C" int kvb_moe_grouped_rows(long long pairs, int experts) {
  const long long mean = experts > 0 ? pairs / experts : pairs;
  return mean <= 48 ? 64 : mean <= 100 ? 128 : 256;
}

// a [rows, K] (the pairs' rows, expert by expert), w [E, weight_rows, K], out [rows, width]; tiles and meta from
// kvb_moe_align with row tiles of `tile_rows`.
extern "C" int kvb_moe_grouped(void* out, const void* a, const void* w, const int* tiles, const int* meta, long long rows, int E,
                               int width, int K, int tile_rows, int mode, float alpha, float limit, float shift,
                               cudaStream_t stream) {
  if (rows == 0 || E == 0) return 0;
  KVB_REQUIRE(width > 0 && K > 0 && K % 8 == 0 && aligned16(a) && aligned16(w) && aligned16(tiles), "moe_grouped: unsupported sizes or addresses");
  KVB_REQUIRE(mode >= 0 && mode <= 3, "moe_grouped: unknown mode");
  KVB_REQUIRE(rows < (1ll << 31) && (long long)E * 2 * width < (1ll << 31), "moe_grouped: too many rows");
  KvbEncodeTiledFn encode = kvb_encode_tiled_fn();
  KVB_REQUIRE(encode != nullptr, "moe_grouped: the driver does not export cuTensorMapEncodeTiled");
  const bool joined = mode == MG_SILU || mode == MG_CLAMPED;
  GroupedParams p = {};
  p.out = (bf16*)out;
  p.tiles = (const int4*)tiles;
  p.meta = meta;
  p.width = width;
  p.weight_rows = joined ? 2 * width : width;
  p.second = joined ? width : 128;
  p.weight_tiles = joined ? (width + 127) / 128 : (width + 255) / 256;
  p.k_stages = (K + MG_K - 1) / MG_K;
  p.alpha = alpha; p.limit = limit; p.shift = shift;
  p.status = kvb_status_word();
  KVB_REQUIRE(p.status != nullptr, "moe_grouped: no status word");
  alignas(64) CUtensorMap w_map, a_map;
  const cuuint64_t strides[1] = {(cuuint64_t)K * sizeof(bf16)};
  const cuuint32_t elem[2] = {1, 1};
  for (int i = 0; i < 2; ++i) {
    const cuuint64_t dims[2] = {(cuuint64_t)K, i == 0 ? (cuuint64_t)E * p.weight_rows : (cuuint64_t)rows};
    const cuuint32_t box[2] = {MG_K, i == 0 ? 128u : 64u};
    KVB_REQUIRE(encode(i == 0 ? &w_map : &a_map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(i == 0 ? w : a), dims, strides, box,
                       elem, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                       CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS,
                "moe_grouped: cuTensorMapEncodeTiled failed");
  }
  const int sms = kvb_sm_count() > 0 ? kvb_sm_count() : 148;
#define KVB_GROUPED(NT, MODE)                                                                                              \
  if (tile_rows == NT && mode == MODE) {                                                                                   \
    KVB_CHECK_CUDA(cudaFuncSetAttribute(moe_grouped_kernel<NT, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize,         \
                                        GroupedRing<NT>::BYTES));                                                          \
    KVB_CHECK_CUDA(kvb_launch((moe_grouped_kernel<NT, MODE>), dim3(sms), dim3(MG_THREADS), GroupedRing<NT>::BYTES, stream, true, \
                              w_map, a_map, p));                                                                           \
    KVB_CHECK_LAUNCH();                                                                                                    \
    return 0;                                                                                                              \
  }
#define KVB_GROUPED_MODES(NT) KVB_GROUPED(NT, MG_SILU) KVB_GROUPED(NT, MG_CLAMPED) KVB_GROUPED(NT, MG_SQUARED) KVB_GROUPED(NT, MG_PLAIN)
  KVB_GROUPED_MODES(64) KVB_GROUPED_MODES(128) KVB_GROUPED_MODES(256)
#undef KVB_GROUPED_MODES
#undef KVB_GROUPED
  return kvb_fail(-1, "moe_grouped: tiles of 64, 128 or 256 rows", __FILE__, __LINE__);
}

KVB_TRACE_TU(moe_tc5)
