// Grouped products of a mixture of experts for prompts, bf16, on the 5th-generation tensor cores: the (token, expert) pairs'
// rows lie expert by expert (moe_align, moe_gather), and for every row r of expert e
//   first product:   hidden[r, f] = join(gate[e, f] . a[r], up[e, f] . a[r])     or   max(up[e, f] . a[r], 0)^2
//   second product:  out[r, n] = down[e, n] . hidden[r]
// in one launch each, the activation formed from the 32-bit sums.
//
// The experts' rows are few and uneven (256 on average where 2,048 tokens choose 4 of 32 experts), so they are the tensor
// pipe's N, which may be any multiple of 32 up to 256, and the weights its M: two blocks on neighbouring SMs multiply 256
// weight rows, 128 each (and, with gated units, the 256 rows of the other matrix beside them), with up to NT rows of one
// expert, half of which lie in either block's shared memory.  An expert's rows are cut into equal tiles (moe_align's table),
// nothing is multiplied that is not there but a run's last few rows up to 32, and the host need not know the experts' loads.
//
// One pair of blocks a pair of SMs; the pairs take (expert, weight tile, row tile) in turn, the row tiles of a weight tile next
// to one another so that weights come from memory once.  In each block warp 0 brings its weight rows and warp 2 its half of
// the expert's rows by TMA, 64 k a stage, all of it reported to block 0; warp 1 of block 0 issues the products; the other 16 warps
// take the block's accumulators out of tensor memory and join them (a lane owns a weight row), turn 16 rows of 32 results in
// shared memory and store them in pieces of 16 bytes.  The ring runs on from item to item; where tensor memory holds them, two sets of accumulators
// alternate.
//
// What bounds it: with many rows the tensor pipe at the clock that the power limit leaves (72 to 78 % of its cycles; the rest is the
// joining of gated units, 256 rows of which fill tensor memory, and pairs of blocks that have one item fewer); with few the
// passes over the weights.  32 experts of 3,584 at width 4,096, 4 a token, whole call with the choices given (B200, call after
// call, beside two batched library products at a common stride and an activation between): 2,048 tokens 706 us and 837; 1,000
// tokens 516 and 628; 130 tokens 446 and 522 (430 of bytes); 16 experts of 4,096 at width 2,048, 2 a token: 2,048 tokens 236
// and 287, 260 tokens 146 and 197.  Single blocks with tiles of 128 x 256 took 763 of 878; one lane alone asking for the copies
// (90 cycles each) 850; results stored by lanes, two bytes each, by eight warps 766; items taken from a counter instead of in
// turn 747 of 860.
#include <cuda.h>
#include <string.h>

#include "common.cuh"
#include "sm100.cuh"

#define MG_K 64
#define MG_W_BYTES (128 * MG_K * 2)         // a block's 128 weight rows of a stage
#define MG_OUT_WARPS 16
#define MG_OUT_BYTES 1024                   // a warp's 16 rows of 32 results on their way out
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
  int weight_rows, second;                  // rows of an expert's matrix; the up rows' distance from the gate rows
  int weight_tiles, k_stages;
  int out16;                                // rows of out are whole 16-byte pieces
  float alpha, limit, shift;
  int* status;
};

template <int NT, bool JOINED> struct GroupedRing {
  static constexpr int WEIGHTS = JOINED ? 2 : 1;
  static constexpr int BOX = NT / 2 < 64 ? NT / 2 : 64;               // rows of a copy of the experts' rows
  static_assert(NT / 2 % BOX == 0, "a block's half of the rows is whole copies: none goes beyond its place");
  static constexpr int STAGE = WEIGHTS * MG_W_BYTES + NT / 2 * MG_K * 2;
  static constexpr int ROOM = 226 * 1024 - MG_OUT_WARPS * MG_OUT_BYTES;
  static constexpr int STAGES = ROOM / STAGE < 8 ? ROOM / STAGE : 8;
  static constexpr int BUFFERS = WEIGHTS * NT > 256 ? 1 : 2;          // sets of accumulators
  static constexpr int BYTES = STAGES * STAGE + MG_OUT_WARPS * MG_OUT_BYTES + 256;
};

__device__ __forceinline__ void mg_ld16(unsigned taddr, float (&v)[16]) {
  unsigned* r = reinterpret_cast<unsigned*>(v);
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                 "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]) : "r"(taddr));
}

template <int NT, int MODE>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(MG_THREADS, 1)
moe_grouped_kernel(const __grid_constant__ CUtensorMap w_map, const __grid_constant__ CUtensorMap a_map, const GroupedParams p) {
  constexpr bool JOINED = MODE == MG_SILU || MODE == MG_CLAMPED;
  using Ring = GroupedRing<NT, JOINED>;
  constexpr int STAGES = Ring::STAGES, BUFFERS = Ring::BUFFERS, WEIGHTS = Ring::WEIGHTS, BOX = Ring::BOX;
  KVB_KERNEL_PROLOGUE(KVB_TAG_MOE_GEMM);
  extern __shared__ __align__(1024) unsigned char mg_dyn[];
  unsigned char* out_smem = mg_dyn + STAGES * Ring::STAGE;
  unsigned long long* full = reinterpret_cast<unsigned long long*>(out_smem + MG_OUT_WARPS * MG_OUT_BYTES);   // block 0's counts
  unsigned long long* empty = full + STAGES;
  unsigned long long* acc_full = empty + STAGES;             // [BUFFERS]
  unsigned long long* acc_empty = acc_full + BUFFERS;        // [BUFFERS] block 0's: the warps of both that take them out
  unsigned long long* drain = acc_empty + BUFFERS;           // given up: products in flight
  unsigned* tmem_slot = reinterpret_cast<unsigned*>(drain + 1);
  int* abort_flag = reinterpret_cast<int*>(tmem_slot + 1);
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const unsigned rank = kvb_cluster_rank();
  const int pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) { kvb_mbar_init(&full[s], 1); kvb_mbar_init(&empty[s], 1); }
    for (int b = 0; b < BUFFERS; ++b) { kvb_mbar_init(&acc_full[b], 1); kvb_mbar_init(&acc_empty[b], 2 * MG_OUT_WARPS); }
    kvb_mbar_init(drain, 1);
    *abort_flag = (kvb_smem(mg_dyn) & 1023u) ? 1 : 0;        // cannot happen with the alignment asked for; never run misaligned
    kvb_mbar_init_fence();
  }
  if (warp == 1) kvb_tc5_alloc_pair(tmem_slot, 512u);
  kvb_tc5_fence_before();
  kvb_cluster_sync();                                        // both blocks' barriers stand
  kvb_tc5_fence_after();
  const unsigned tmem = __shfl_sync(0xffffffffu, *tmem_slot, 0);
  auto gave_up = [&] {
    atomicOr(p.status, KVB_STATUS_WAIT_TIMEOUT);
    atomicExch(abort_flag, 1);
  };
  auto aborted = [&] { return *reinterpret_cast<volatile int*>(abort_flag) != 0; };

  const int items = p.meta[1] * p.weight_tiles;
  struct Item { int expert, row0, rows, tile, half; };       // half: rows of the product that each block holds
  auto item = [&](int i) {
    Item it;
    const int4 any = p.tiles[i / p.weight_tiles];            // a row tile of the item's expert
    const int count = any.z >> 12, r = i - any.w * p.weight_tiles;
    it.tile = r / count;
    const int4 mine = p.tiles[any.w + r - it.tile * count];
    it.expert = mine.x;
    it.row0 = mine.y;
    it.rows = mine.z & 0xfff;
    it.half = (it.rows + 31) / 32 * 16;
    return it;
  };

  if (warp == 0 || warp == 2) {
    // ================= weights (warp 0) and rows (warp 2): whole warps, one lane issues =================
    const unsigned leader = kvb_elect(), ring = kvb_smem(mg_dyn) + (warp == 0 ? 0 : WEIGHTS * MG_W_BYTES);
    const unsigned bar0 = kvb_cluster_addr(full, 0), first = rank == 0 && warp == 0 ? leader : 0u;
    unsigned at = 0;                                         // stages asked for so far
    bool ok = true;
    for (int i = pair; i < items && ok; i += pairs) {
      const Item it = item(i);
      const int boxes = __shfl_sync(0xffffffffu, (it.half + BOX - 1) / BOX, 0);
      const int row = __shfl_sync(0xffffffffu, warp == 0 ? it.expert * p.weight_rows + it.tile * 256 + (int)rank * 128
                                                         : it.row0 + (int)rank * it.half, 0);
      const unsigned bytes = WEIGHTS * MG_W_BYTES + boxes * BOX * MG_K * 2;
      for (int k = 0; k < p.k_stages; ++k, ++at) {
        const unsigned s = at % STAGES;
        if (at >= STAGES) ok = __all_sync(0xffffffffu, kvb_mbar_wait<MG_SPIN_LIMIT, 4096>(&empty[s], ((at / STAGES) - 1) & 1));
        if (!ok) break;
        const unsigned to = ring + s * Ring::STAGE, bar = bar0 + s * 8;
        if (warp == 0) {
          if (first) kvb_mbar_expect_tx(&full[s], 2 * bytes);          // both blocks'
          kvb_tma_2d_pair(to, &w_map, k * MG_K, row, bar, leader);
          if (JOINED) kvb_tma_2d_pair(to + MG_W_BYTES, &w_map, k * MG_K, row + p.second, bar, leader);
        } else {
          for (int b = 0; b < boxes; ++b)
            kvb_tma_2d_pair(to + b * BOX * MG_K * 2, &a_map, k * MG_K, row + BOX * b, bar, leader);
        }
      }
    }
    if (!ok) {
      if (lane == 0) gave_up();
      // the copies in flight land before the block may exit: block 0 sees them; block 1 gives them a millisecond
      if (rank == 0)
        for (unsigned j = at < STAGES ? 0 : at - STAGES; j < at; ++j) kvb_mbar_wait<MG_SPIN_LIMIT / 16, 4096>(&full[j % STAGES], (j / STAGES) & 1);
      for (int j = 0; j < 1000; ++j) __nanosleep(1000);
    }
    __syncwarp();
  } else if (warp == 1) {
    // ================= products: block 0's whole warp, one lane issues =================
    if (rank == 0) {
      const unsigned leader = kvb_elect();
      const unsigned long long base = kvb_tc5_desc(kvb_smem(mg_dyn), 16, 1024);
      unsigned at = 0, n = 0;
      bool ok = true;
      for (int i = pair; i < items && ok; i += pairs, ++n) {
        const int half = __shfl_sync(0xffffffffu, item(i).half, 0);
        const unsigned idesc = kvb_tc5_idesc(256, 2 * half, false);
        const unsigned b = n % BUFFERS, acc = tmem + b * WEIGHTS * NT;
        if (n >= BUFFERS) ok = __all_sync(0xffffffffu, kvb_mbar_wait<MG_SPIN_LIMIT, 4096>(&acc_empty[b], ((n / BUFFERS) - 1) & 1));
        for (int k = 0; k < p.k_stages && ok; ++k, ++at) {
          const unsigned s = at % STAGES;
          ok = __all_sync(0xffffffffu, kvb_mbar_wait<MG_SPIN_LIMIT, 4096>(&full[s], (at / STAGES) & 1)) && !aborted();
          if (!ok) break;
          kvb_tc5_fence_after();
          const unsigned long long w = base + s * (Ring::STAGE / 16), a = w + WEIGHTS * MG_W_BYTES / 16;
#pragma unroll
          for (int j = 0; j < 4; ++j) {                      // 16 k: 32 bytes of a row of 128
            kvb_tc5_mma_pair(acc, w + 2 * j, a + 2 * j, idesc, k > 0 || j > 0 ? 1u : 0u, leader);
            if (JOINED) kvb_tc5_mma_pair(acc + NT, w + MG_W_BYTES / 16 + 2 * j, a + 2 * j, idesc, k > 0 || j > 0 ? 1u : 0u, leader);
          }
          kvb_tc5_commit_pair(&empty[s], leader);
        }
        if (ok) kvb_tc5_commit_pair(&acc_full[b], leader);
      }
      if (!ok) {
        if (lane == 0) gave_up();
        kvb_tc5_commit_pair(drain, leader);                  // tensor memory is given back below: products in flight first
        kvb_mbar_wait<MG_SPIN_LIMIT, 4096>(drain, 0);
      }
      __syncwarp();
    }
  } else if (warp >= 4) {
    // ================= results: 16 rows at a time, turn about between the four warps of a lane quarter =================
    const int quarter = warp & 3, turn = (warp - 4) >> 2;
    const unsigned lanes = (unsigned)(quarter * 32) << 16;
    unsigned n = 0;
    bool ok = true;
    for (int i = pair; i < items; i += pairs, ++n) {
      const Item it = item(i);
      const unsigned b = n % BUFFERS;
      ok = __all_sync(0xffffffffu, kvb_mbar_wait<MG_SPIN_LIMIT, 4096>(&acc_full[b], (n / BUFFERS) & 1)) && !aborted();
      if (!ok) break;
      kvb_tc5_fence_after();
      const unsigned acc = tmem + lanes + b * WEIGHTS * NT;
      const int feature0 = it.tile * 256 + (int)rank * 128 + quarter * 32;
      bf16* const mine = reinterpret_cast<bf16*>(out_smem + (warp - 4) * MG_OUT_BYTES);
      for (int c = turn * 16; c < it.rows; c += 4 * MG_OUT_WARPS) {
        float u[16], v[16];
        mg_ld16(acc + c, u);
        if (JOINED) mg_ld16(acc + NT + c, v);
        kvb_tc5_wait_ld();
        __syncwarp();                                        // the rows in front have left
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          float r = u[j];
          if (MODE == MG_SILU) {
            r = kvb_silu_for_bf16(u[j]) * v[j];
          } else if (MODE == MG_CLAMPED) {
            const float g = fminf(u[j], p.limit);
            r = __fdividef(g, 1.0f + __expf(-p.alpha * g)) * (fminf(fmaxf(v[j], -p.limit), p.limit) + p.shift);
          } else if (MODE == MG_SQUARED) {
            r = fmaxf(u[j], 0.0f);
            r *= r;
          }
          mine[j * 32 + lane] = __float2bfloat16_rn(r);
        }
        __syncwarp();
        if (p.out16) {
#pragma unroll
          for (int h = 0; h < 2; ++h) {                      // eight rows, four lanes a row
            const int row = h * 8 + (lane >> 2), at = (lane & 3) * 8;
            if (feature0 + at < p.width)
              *reinterpret_cast<uint4*>(p.out + (long long)(it.row0 + c + row) * p.width + feature0 + at) =
                  *reinterpret_cast<const uint4*>(mine + row * 32 + at);
          }
        } else if (feature0 + lane < p.width) {
          for (int j = 0; j < 16; ++j) p.out[(long long)(it.row0 + c + j) * p.width + feature0 + lane] = mine[j * 32 + lane];
        }
      }
      kvb_tc5_fence_before();
      __syncwarp();
      if (lane == 0) kvb_cluster_arrive(kvb_cluster_addr(&acc_empty[b], 0));
    }
    if (!ok && lane == 0) gave_up();
    __syncwarp();
  }
  kvb_tc5_fence_before();
  __syncthreads();
  kvb_cluster_sync();                                        // nobody reads the other's shared memory or tensor memory any more
  if (warp == 1) {
    kvb_tc5_fence_after();
    kvb_tc5_dealloc_pair(tmem, 512u);
  }
}

// Rows of a tile for a batch: `pairs` of `experts`.  Also what moe_align cuts runs by.  Smaller tiles leave room for more stages,
// which keep more of the weights in flight where the rows are few; larger ones pass over the weights less often.  Microseconds
// with tiles of 64, 128 and 256 rows, 32 experts of 3,584 at width 4,096: 24 rows an expert 461, 460, 481; 48: 472, 473, 497; 64:
// 514, 479, 525; 100: 655, 521, 551; 128: 832, 613, 579; 192: 982, 717, 646; 256: 1337, 799, 831; 384: 1563, 1013, 1413 (a second
// tile of few rows an expert); 16 of 4,096 at 2,048: 48: 183, 183, 196; 100: 180, 166, 172; 160: 252, 206, 195; 384: 435, 298, 294.
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
  KVB_REQUIRE(tile_rows == 64 || tile_rows == 128 || tile_rows == 256, "moe_grouped: tiles of 64, 128 or 256 rows");
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
  p.second = width;
  p.weight_tiles = (width + 255) / 256;
  p.k_stages = (K + MG_K - 1) / MG_K;
  p.out16 = width % 8 == 0 && aligned16(out) ? 1 : 0;
  p.alpha = alpha; p.limit = limit; p.shift = shift;
  p.status = kvb_status_word();
  KVB_REQUIRE(p.status != nullptr, "moe_grouped: no status word");
  alignas(64) CUtensorMap w_map, a_map;
  const cuuint64_t strides[1] = {(cuuint64_t)K * sizeof(bf16)};
  const cuuint32_t elem[2] = {1, 1};
  for (int i = 0; i < 2; ++i) {
    const cuuint64_t dims[2] = {(cuuint64_t)K, i == 0 ? (cuuint64_t)E * p.weight_rows : (cuuint64_t)rows};
    const cuuint32_t box[2] = {MG_K, i == 0 ? 128u : tile_rows / 2 < 64 ? (cuuint32_t)tile_rows / 2 : 64u};
    KVB_REQUIRE(encode(i == 0 ? &w_map : &a_map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(i == 0 ? w : a), dims, strides, box,
                       elem, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                       CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS,
                "moe_grouped: cuTensorMapEncodeTiled failed");
  }
  const int sms = kvb_sm_count() > 0 ? kvb_sm_count() : 148;
#define KVB_GROUPED(NT, MODE)                                                                                              \
  if (tile_rows == NT && mode == MODE) {                                                                                   \
    constexpr int bytes = GroupedRing<NT, MODE == MG_SILU || MODE == MG_CLAMPED>::BYTES;                                   \
    KVB_CHECK_CUDA(cudaFuncSetAttribute(moe_grouped_kernel<NT, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes)); \
    KVB_CHECK_CUDA(kvb_launch((moe_grouped_kernel<NT, MODE>), dim3(sms / 2 * 2), dim3(MG_THREADS), bytes, stream, true,    \
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
