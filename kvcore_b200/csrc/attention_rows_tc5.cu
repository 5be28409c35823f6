// Flash attention for prompt portions on the 5th-generation tensor cores when keys are 128 or 192 entries wide and values
// a multiple of 128, both anywhere in the rows of a plane: the form of attention_prefill_tc5.cu for the mixers of
// attention_flash_dims.cu (several score maps a value head, 32-bit results, a sink per query head, a slope per query head
// times the distance taken off the score).  bf16 operands, 32-bit scores, softmax and accumulation.
//
// A block owns two tiles of 128 query rows of one (request, key head, slice of 128 value columns), A and B (A alone in
// launches of few blocks: kvb_tc5_query_tiles); a row is a
// (token, query head of the key head's group) pair.  It walks the keys in tiles of 128; eleven warps as there: two softmax
// warpgroups (a thread a row), a producer warp for keys and one for values, one thread that issues the products
//     S_A(0), S_B(0); per key tile j:  O_A += P_A(j).V(j), S_A(j+1), O_B += P_B(j).V(j), S_B(j+1).
// Behind a window B begins with the first key tile that it sees itself, so that a row's result has the same bits in blocks
// of one and of two query tiles.
// Keys are staged as KH parts of 64 columns (128-byte swizzle), two stages; values as two parts, in two stages beside keys
// of 128, in one beside keys of 192 (the shared memory is then full: 96 KB of queries, 96 of keys, 32 of values; the next
// values are asked for when B's product with the last ones has been taken, half a key tile's time ahead of A's).
// Rows come by TMA, a box a page; or, when the rows of a request's positions lie one behind the other (keys carried up
// from cached latents), a box of 128 rows that may begin in front of the request's first row and end behind its last.
// Rows that nobody in the block sees are another request's, or what a page's former owner left there: their scores are
// masked, and their values, which a probability of zero would not undo if they were no numbers, are cleared in shared
// memory ahead of the product (pages that hold nothing but such rows are not read at all).
// Weights go in as two bf16, the second what the first rounding left: the products are exact to 2^-18 of a weight, the row
// sum is taken in 32 bits, and the maximum may lag behind (see below).  With one bf16 and that lag, rows that a few large
// weights decide were up to 1.6 times as far from their values in 64 bits as the mma.sync tiles of attention_flash_dims.cu
// leave them, whose running maximum makes the largest weights exact: 2,048 tokens with scores up to 15, 9.8e-4 of the result
// and 6.1e-4; now 5e-6.
// What bounds it is the chain of products and softmax of each query tile (see attention_prefill_tc5.cu), not a unit.
// One prompt of 2,048 tokens, call by call (B200; in brackets what the weights' second half costs of it, and the mma.sync
// tiles): carried-up latents, 32 heads of 192 / 128: 111 us (15; 394); 16 heads of two maps, 128 / 256: 179 us (29; 432);
// 32 heads over 8, 128 / 128, window 1,024, a sink: 118 us (12; 245), with slopes 135 (19; 245).  Few rows as well: 40 tokens
// behind 2,000: 89 us (10; 188).
//
// Tensor memory: 512 columns = S_A | S_B | O_A | O_B of 128 each; P_X lies over S_X, the second halves in the last 64 columns.
// Every wait is bounded: on a time-out the thread sets the WAIT_TIMEOUT status bit, the block drains, frees its tensor
// memory and returns.
#include <cuda.h>
#include <string.h>

#include "common.cuh"
#include "sm100.cuh"

#define RT_BM 128
#define RT_BN 128
#define RT_V 128                          // value columns of a block
#define RT_THREADS 352
#define RT_SPIN_LIMIT (1u << 20)
#define RT_PART_BYTES (128 * 128)         // 64 columns of 128 rows
#define RT_WAIT(bar, parity) kvb_mbar_wait<RT_SPIN_LIMIT, 4096>(bar, parity)

struct RowsTc5Params {
  void* out; long long out_token, out_head; int out_f32;
  const bf16* q; long long q_token, q_head;
  const int* table; int table_stride;
  const int* query_start; const int* context_lens;
  int G, maps, slices, page_rows, num_pages, window, in_order;
  int k_head, v_head;                     // columns between two heads of a key (value) row
  float scale_log2;
  const float* sink; const float* slopes;
  int* status;
  int q_by_tma;
  int tiles;                              // query tiles of a block (kvb_tc5_query_tiles)
  int no_row;                             // behind the last row of the planes: a box there is all zeros
};

// Byte offset of the 16-byte piece `piece` of row `r` in an operand tile stored as swizzled parts of 64 columns.
__device__ __forceinline__ unsigned rt_piece_off(int r, int piece) {
  return (unsigned)((piece >> 3) * RT_PART_BYTES + r * 128 + (((piece & 7) ^ (r & 7)) << 4));
}
__device__ __forceinline__ float rt_max3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}
// (d0, d1) = (a0, a1) * b + c
__device__ __forceinline__ void rt_fma2(float& d0, float& d1, float a0, float a1, float b, float c) {
  asm("{.reg .b64 ra, rb, rc, rd;\n mov.b64 ra, {%2, %3};\n mov.b64 rb, {%4, %4};\n mov.b64 rc, {%5, %5};\n"
      " fma.rn.f32x2 rd, ra, rb, rc;\n mov.b64 {%0, %1}, rd;}\n"
      : "=f"(d0), "=f"(d1) : "f"(a0), "f"(a1), "f"(b), "f"(c));
}
__device__ __forceinline__ void rt_add2(float& s0, float& s1, float a0, float a1) {
  asm("{.reg .b64 ra, rb, rd;\n mov.b64 ra, {%0, %1};\n mov.b64 rb, {%2, %3};\n add.rn.f32x2 rd, ra, rb;\n"
      " mov.b64 {%0, %1}, rd;}\n"
      : "+f"(s0), "+f"(s1) : "f"(a0), "f"(a1));
}
// (h0, h1) and what they are short of (e0, e1): exact, since h is e rounded
__device__ __forceinline__ void rt_short_of(float& d0, float& d1, float e0, float e1, float h0, float h1) {
  asm("{.reg .b64 rh, rm, re, rd;\n mov.b64 rh, {%4, %5};\n mov.b64 rm, {%6, %6};\n mov.b64 re, {%2, %3};\n"
      " fma.rn.f32x2 rd, rh, rm, re;\n mov.b64 {%0, %1}, rd;}\n"
      : "=f"(d0), "=f"(d1) : "f"(e0), "f"(e1), "f"(h0), "f"(h1), "f"(-1.0f));
}
// (lo, hi) rounded to two bf16 in one register, the lower key in the lower half, and back.
__device__ __forceinline__ float rt_pack(float lo, float hi) {
  unsigned d;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(hi), "f"(lo));
  return __uint_as_float(d);
}
__device__ __forceinline__ float rt_low(float pack) { return __uint_as_float(__float_as_uint(pack) << 16); }
__device__ __forceinline__ float rt_high(float pack) { return __uint_as_float(__float_as_uint(pack) & 0xffff0000u); }

// KH: parts of 64 columns of a key.  SLOPE: slopes are given.
template <int KH, bool SLOPE>
__global__ void __launch_bounds__(RT_THREADS, 1)
flash_rows_tc5_kernel(const __grid_constant__ CUtensorMap k_map, const __grid_constant__ CUtensorMap v_map,
                      const __grid_constant__ CUtensorMap q_map, const RowsTc5Params p) {
  KVB_KERNEL_PROLOGUE(KVB_TAG_FLASH_DIMS);
  constexpr unsigned K_BYTES = KH * RT_PART_BYTES, V_BYTES = 2 * RT_PART_BYTES;
  constexpr int VS = KH == 2 ? 2 : 1;                       // stages of values
  extern __shared__ __align__(1024) unsigned char rt_dyn[];
  unsigned char* q_smem = rt_dyn;                            // tile A, tile B
  unsigned char* k_smem = q_smem + 2 * K_BYTES;              // 2 stages
  unsigned char* v_smem = k_smem + 2 * K_BYTES;              // VS stages
  unsigned long long* bars = reinterpret_cast<unsigned long long*>(v_smem + VS * V_BYTES);
  unsigned long long* k_full = bars;        // [2 stages]
  unsigned long long* k_empty = bars + 2;   // [2]
  unsigned long long* v_full = bars + 4;    // [VS]
  unsigned long long* v_empty = bars + 6;   // [VS]
  unsigned long long* s_full = bars + 8;    // [2 query tiles]
  unsigned long long* p_ready = bars + 10;  // [2 query tiles]
  unsigned long long* pv_done = bars + 12;  // [2 query tiles]
  unsigned long long* q_full = bars + 14;
  unsigned* tmem_slot = reinterpret_cast<unsigned*>(bars + 15);
  int* abort_flag = reinterpret_cast<int*>(tmem_slot + 1);

  // later query tiles see more keys: they are handed out first
  const int req = blockIdx.y, kh = blockIdx.x / p.slices, slice = blockIdx.x % p.slices;
  const int vh = kh / p.maps, map = kh % p.maps, pair = gridDim.z - 1 - blockIdx.z;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int q_begin = p.query_start[req];
  const int q_len = p.query_start[req + 1] - q_begin;
  const int context = p.context_lens[req];
  const int rows_total = q_len * p.G;
  const int row0 = pair * p.tiles * RT_BM;
  if (row0 >= rows_total) return;           // whole block, before any barrier or allocation
  if (kvb_smem(rt_dyn) & 1023u) {            // cannot happen with the alignment asked for; never run misaligned
    if (threadIdx.x == 0) atomicOr(p.status, KVB_STATUS_WAIT_TIMEOUT);
    return;
  }
  const bool has_b = p.tiles == 2 && row0 + RT_BM < rows_total;
  const int last_row_a = min(row0 + RT_BM, rows_total) - 1;
  const int last_row_b = min(row0 + 2 * RT_BM, rows_total) - 1;
  const int first_pos_a = context + row0 / p.G;
  const int key_lo = p.window > 0 ? max(0, first_pos_a - p.window + 1) : 0;
  const int tile_begin = key_lo / RT_BN;
  const int n_a = (context + last_row_a / p.G + RT_BN) / RT_BN - tile_begin;              // >= 1
  const int n_b = has_b ? (context + last_row_b / p.G + RT_BN) / RT_BN - tile_begin : 0;  // >= n_a when tile B exists
  const int num_tiles = max(n_a, n_b);
  // the first key tile that B sees (A's is 0); its own tiles are counted from there
  const int b_begin = has_b && p.window > 0 ? max(0, context + (row0 + RT_BM) / p.G - p.window + 1) / RT_BN - tile_begin : 0;
  const int key_hi = context + (has_b ? last_row_b : last_row_a) / p.G + 1;
  auto query_head = [&](int flat) { return (vh * p.G + flat % p.G) * p.maps + map; };

  if (threadIdx.x < 15) {
    kvb_mbar_init(&bars[threadIdx.x], (threadIdx.x == 10 || threadIdx.x == 11) ? 128u : 1u);
    if (threadIdx.x == 0) *abort_flag = 0;
    kvb_mbar_init_fence();
  }
  if (warp == 8 && lane < 3) {
    const CUtensorMap* which = lane == 0 ? &k_map : lane == 1 ? &v_map : &q_map;
    if (lane < 2 || p.q_by_tma)
      asm volatile("prefetch.tensormap [%0];\n" ::"l"(reinterpret_cast<unsigned long long>(which)) : "memory");
  }
  if (warp == 10) kvb_tc5_alloc(tmem_slot, 512u);
  if (warp < 8 && !p.q_by_tma) {             // thread t of warpgroup X: row t of tile X
    const int r = threadIdx.x & 127, x = threadIdx.x >> 7;
    const int flat = row0 + x * RT_BM + r;
    const bool valid = flat < rows_total && x < p.tiles;
    const bf16* src = p.q + (size_t)(q_begin + (valid ? flat / p.G : 0)) * p.q_token + (size_t)query_head(valid ? flat : 0) * p.q_head;
    unsigned char* dst = q_smem + x * K_BYTES;
#pragma unroll
    for (int c = 0; c < KH * 8; ++c) {
      uint4 v = make_uint4(0, 0, 0, 0);
      if (valid) v = *reinterpret_cast<const uint4*>(src + c * 8);
      *reinterpret_cast<uint4*>(dst + rt_piece_off(r, c)) = v;
    }
    kvb_fence_async_shared();                // generic writes -> visible to the products' reads
  }
  // rows of the copies: a batch of 32 looked up at a time, a batch ahead
  const int* entries = p.table + (size_t)req * p.table_stride;
  const int ppt = RT_BN / p.page_rows;       // copies a tile (and part): 1 or 2..16
  const int total_entries = num_tiles * ppt;
  auto fetch = [&](int entry) -> int {
    if (entry >= total_entries) return p.no_row;
    if (p.in_order) {                        // an entry is a tile: its first row, counted back from the first that is seen
      const int key0 = (tile_begin + entry) * RT_BN, key = max(key0, key_lo);
      if (key >= key_hi || key >= p.table_stride) return p.no_row;
      const int row = entries[key];
      if (row <= 0 || row >= p.num_pages) {
        atomicOr(p.status, KVB_STATUS_BAD_PAGE);
        return p.no_row;
      }
      return row - (key - key0);
    }
    const int index = tile_begin * ppt + entry;
    if (index >= p.table_stride || index * p.page_rows >= key_hi || (index + 1) * p.page_rows <= key_lo) return p.no_row;
    const int page = entries[index];
    if (page < 0 || page >= p.num_pages) atomicOr(p.status, KVB_STATUS_BAD_PAGE);
    return page > 0 && page < p.num_pages ? page * p.page_rows : p.no_row;      // page 0 is nobody's
  };
  int cur = 0, nxt = 0;
  if (warp == 8 || warp == 9) {
    cur = fetch(lane);
    nxt = fetch(32 + lane);
  }
  kvb_tc5_fence_before();
  __syncthreads();
  kvb_tc5_fence_after();
  const unsigned tmem_base = *tmem_slot;

  if (warp == 8 || warp == 9) {
    // ================= producers: warp 8 brings keys, warp 9 values =================
    const bool is_k = warp == 8;
    const CUtensorMap* from = is_k ? &k_map : &v_map;
    unsigned char* ring = is_k ? k_smem : v_smem;
    unsigned long long* full = is_k ? k_full : v_full;
    unsigned long long* empty = is_k ? k_empty : v_empty;
    const int stages = is_k ? 2 : VS, parts = is_k ? KH : 2;
    const unsigned bytes = is_k ? K_BYTES : V_BYTES;
    const int column = is_k ? kh * p.k_head : vh * p.v_head + slice * RT_V;
    if (is_k && lane == 0 && p.q_by_tma) {   // rows in (token, head of the group) order; tokens beyond the batch as zeros
      const int token0 = q_begin + row0 / p.G;
      kvb_mbar_expect_tx(q_full, (has_b ? 2u : 1u) * K_BYTES);
      for (int x = 0; x < (has_b ? 2 : 1); ++x)
        for (int part = 0; part < KH; ++part)
          kvb_tma_4d(q_smem + x * K_BYTES + part * RT_PART_BYTES, &q_map, part * 64, 0, kh, token0 + x * (RT_BM / p.G), q_full);
    }
    int issued = 0;
    for (int j = 0; j < num_tiles; ++j) {
      const int s = j % stages, turn = j / stages;
      const int e0 = j * ppt;
      if (e0 > 0 && (e0 & 31) == 0) {
        cur = nxt;
        nxt = fetch(e0 + 32 + lane);
      }
      const int row = __shfl_sync(0xffffffffu, cur, (e0 + lane) & 31);
      int ok = 1;
      if (lane == 0) {
        if (j >= stages && !RT_WAIT(&empty[s], (turn - 1) & 1)) ok = 0;
        if (ok && *reinterpret_cast<volatile int*>(abort_flag)) ok = 0;
        if (ok) kvb_mbar_expect_tx(&full[s], bytes);
      }
      ok = __shfl_sync(0xffffffffu, ok, 0);
      if (!ok) break;
      if (lane < ppt) {
        unsigned char* dst = ring + s * bytes + lane * p.page_rows * 128;
        for (int part = 0; part < parts; ++part)
          kvb_tma_2d(dst + part * RT_PART_BYTES, from, column + part * 64, row, &full[s]);
      }
      issued = j + 1;
    }
    if (lane == 0 && issued < num_tiles) {
      atomicOr(p.status, KVB_STATUS_WAIT_TIMEOUT);
      atomicExch(abort_flag, 1);
    }
    if (lane == 0 && *reinterpret_cast<volatile int*>(abort_flag)) {
      // let the copies that were issued land before the block may exit
      for (int j = max(0, issued - stages); j < issued; ++j) RT_WAIT(&full[j % stages], (j / stages) & 1);
      if (is_k && p.q_by_tma) RT_WAIT(q_full, 0);
    }
  } else if (warp == 10) {
    // ================= the issuing thread =================
    if (lane == 0) {
      const unsigned idesc_s = kvb_tc5_idesc(RT_BM, RT_BN, false);   // A, B both K-major
      const unsigned idesc_pv = kvb_tc5_idesc(RT_BM, RT_V, true);    // B (the values) MN-major
      bool ok = true;
      // descriptors of a tile differ from step to step in their address field alone: made once, a step adds a constant
      const unsigned long long q_desc[2] = {kvb_tc5_desc(kvb_smem(q_smem), 16, 1024), kvb_tc5_desc(kvb_smem(q_smem + K_BYTES), 16, 1024)};
      const unsigned long long k_desc[2] = {kvb_tc5_desc(kvb_smem(k_smem), 16, 1024), kvb_tc5_desc(kvb_smem(k_smem + K_BYTES), 16, 1024)};
      const unsigned long long v_desc[2] = {kvb_tc5_desc(kvb_smem(v_smem), RT_PART_BYTES, 1024),
                                            kvb_tc5_desc(kvb_smem(v_smem + (VS - 1) * V_BYTES), RT_PART_BYTES, 1024)};
      constexpr int PART16 = RT_PART_BYTES >> 4;
      auto issue_s = [&](int x, int st) {
        kvb_tc5_mma8_ss<2, PART16 - 6, 2, PART16 - 6>(tmem_base + x * RT_BN, q_desc[x], k_desc[st], idesc_s, 0u);
        if (KH == 3) kvb_tc5_mma4_ss<2, 2>(tmem_base + x * RT_BN, q_desc[x] + 2 * PART16, k_desc[st] + 2 * PART16, idesc_s);
        kvb_tc5_commit(&s_full[x]);
      };
      auto issue_pv = [&](int x, int st, bool add) {
        kvb_tc5_mma8_ts<8, 128>(tmem_base + 256 + x * RT_V, tmem_base + x * RT_BN, v_desc[st], idesc_pv, add ? 1u : 0u);
        kvb_tc5_mma8_ts<8, 128>(tmem_base + 256 + x * RT_V, tmem_base + x * RT_BN + 64, v_desc[st], idesc_pv, 1u);
        kvb_tc5_commit(&pv_done[x]);
      };
      if (p.q_by_tma && !RT_WAIT(q_full, 0)) ok = false;
      if (ok && !RT_WAIT(&k_full[0], 0)) ok = false;
      if (ok) {
        kvb_tc5_fence_after();
        issue_s(0, 0);
        if (has_b && b_begin == 0) issue_s(1, 0);
        kvb_tc5_commit(&k_empty[0]);
      }
      for (int j = 0; j < num_tiles && ok; ++j) {
        const int vs = j % VS, ks = (j + 1) & 1;
        const bool more = j + 1 < num_tiles;
        if (!RT_WAIT(&v_full[vs], (j / VS) & 1)) { ok = false; break; }
        if (j < n_a) {
          if (!RT_WAIT(&p_ready[0], j & 1)) { ok = false; break; }
          kvb_tc5_fence_after();
          issue_pv(0, vs, j > 0);
        }
        if (more) {
          if (!RT_WAIT(&k_full[ks], ((j + 1) >> 1) & 1)) { ok = false; break; }
          kvb_tc5_fence_after();
          if (j + 1 < n_a) issue_s(0, ks);
        }
        if (j >= b_begin && j < n_b) {
          if (!RT_WAIT(&p_ready[1], (j - b_begin) & 1)) { ok = false; break; }
          kvb_tc5_fence_after();
          issue_pv(1, vs, j > b_begin);
        }
        kvb_tc5_commit(&v_empty[vs]);
        if (more) {
          if (j + 1 >= b_begin && j + 1 < n_b) issue_s(1, ks);
          kvb_tc5_commit(&k_empty[ks]);
        }
      }
      if (!ok) {
        atomicOr(p.status, KVB_STATUS_WAIT_TIMEOUT);
        atomicExch(abort_flag, 1);
      }
    }
  } else {
    // ================= softmax: thread r of warpgroup x owns row r of tile x =================
    const int r = threadIdx.x & 127, x = threadIdx.x >> 7;
    const int begin = x == 0 ? 0 : b_begin, n_mine = (x == 0 ? n_a : n_b) - begin;     // this tile's key tiles
    const int flat = row0 + x * RT_BM + r;
    const bool row_valid = flat < rows_total;
    const int pos = context + (row_valid ? flat / p.G : 0), hq = query_head(row_valid ? flat : 0);
    const int row_lo = p.window > 0 ? max(0, pos - p.window + 1) : 0;
    const int first_pos = context + (row0 + x * RT_BM) / p.G;
    const unsigned lane_addr = ((unsigned)((warp & 3) * 32) << 16);
    const bool ragged = row0 + (x + 1) * RT_BM > rows_total;
    const unsigned s_addr = tmem_base + lane_addr + x * RT_BN;
    const unsigned o_addr = tmem_base + lane_addr + 256 + x * RT_V;
    float row_max = -INFINITY, row_sum = 0.0f;            // row_max in the scaled (log2) domain
    const float slope = SLOPE ? p.slopes[hq] * 1.4426950408889634f : 0.0f;
    const float scale_log2 = SLOPE ? 1.0f : p.scale_log2; // with slopes the scores are brought into the log2 domain first
    bool ok = true;
    for (int turn = 0; turn < n_mine; ++turn) {
      if (!RT_WAIT(&s_full[x], turn & 1)) { ok = false; break; }
      kvb_tc5_fence_after();
      const int j = begin + turn, key0 = (tile_begin + j) * RT_BN;
      const bool need_mask = ragged || p.window > 0 || key0 + RT_BN - 1 > first_pos;
      float s[4][32];
#pragma unroll
      for (int c = 0; c < 4; ++c) kvb_tc5_ld32(s_addr + c * 32, s[c]);
      kvb_tc5_wait_ld();
      if (SLOPE) {
        const float first = slope * (float)(key0 - pos);
#pragma unroll
        for (int c = 0; c < 4; ++c)
#pragma unroll
          for (int i = 0; i < 32; ++i) s[c][i] = fmaf(s[c][i], p.scale_log2, fmaf(slope, (float)(c * 32 + i), first));
      }
      float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
      if (need_mask) {
        const int hi = row_valid ? pos - key0 : -1, lo = row_lo - key0;
        if (p.window > 0) {
#pragma unroll
          for (int c = 0; c < 4; ++c)
#pragma unroll
            for (int i = 0; i < 32; ++i)
              if (c * 32 + i > hi || c * 32 + i < lo) s[c][i] = -INFINITY;
        } else {
#pragma unroll
          for (int c = 0; c < 4; ++c)
#pragma unroll
            for (int i = 0; i < 32; ++i)
              if (c * 32 + i > hi) s[c][i] = -INFINITY;
        }
      }
#pragma unroll
      for (int c = 0; c < 4; ++c)
#pragma unroll
        for (int i = 0; i < 32; i += 2) mx[(i >> 1) & 3] = rt_max3(mx[(i >> 1) & 3], s[c][i], s[c][i + 1]);
      const float tile_max = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])) * scale_log2;   // (the scale is positive); -inf stays -inf
      const float new_max = fmaxf(row_max, tile_max);
      // The maximum is moved (and O rescaled) only when it would grow by more than 2^8.
      const bool grows = new_max > row_max + 8.0f;                       // from -inf too
      const bool move = __any_sync(0xffffffffu, grows);
      float correction = 1.0f;
      if (move) {
        correction = (row_max == -INFINITY) ? 0.0f : exp2f(row_max - new_max);
        row_max = new_max;
      }
      const float shift = (row_max == -INFINITY) ? 0.0f : -row_max;
      float sm[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        float packed[16], rest[16];                  // 32 keys, two bf16 a register
#pragma unroll
        for (int i = 0; i < 32; i += 2) {
          float a0, a1, e0, e1;
          rt_fma2(a0, a1, s[c][i], s[c][i + 1], scale_log2, shift);      // masked entries stay -inf
          asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e0) : "f"(a0));
          asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e1) : "f"(a1));
          rt_add2(sm[i & 2], sm[(i & 2) + 1], e0, e1);
          packed[i / 2] = rt_pack(e0, e1);
          rt_short_of(a0, a1, e0, e1, rt_low(packed[i / 2]), rt_high(packed[i / 2]));
          rest[i / 2] = rt_pack(a0, a1);
        }
        kvb_tc5_st16(s_addr + c * 16, packed);       // over S(j); S(j+1) comes after the tensor pipe has taken P(j)
        kvb_tc5_st16(s_addr + 64 + c * 16, rest);
      }
      row_sum = row_sum * correction + ((sm[0] + sm[1]) + (sm[2] + sm[3]));
      if (move && turn > 0) {                        // P(j-1).V(j-1) has landed: it was issued before S(j)
#pragma unroll 1
        for (int c = 0; c < 4; ++c) {
          float o[32];
          kvb_tc5_ld32(o_addr + c * 32, o);
          kvb_tc5_wait_ld();
#pragma unroll
          for (int i = 0; i < 32; ++i) o[i] *= correction;
          kvb_tc5_st32(o_addr + c * 32, o);
        }
      }
      // Values of rows outside [key_lo, key_hi): thread r clears row r, in the first tile that reads this key tile's
      // values (A where it sees the tile), whose product waits for all its threads and is issued ahead of the other's.
      // (A warp with such rows waits and goes on as a whole: the tensor memory's instructions behind are the whole warp's.)
      const bool nobodys = key0 + r < key_lo || key0 + r >= key_hi;
      if ((j < n_a) == (x == 0) && __any_sync(0xffffffffu, nobodys)) {
        const int vs = j % VS;
        if (!__all_sync(0xffffffffu, RT_WAIT(&v_full[vs], (j / VS) & 1))) { ok = false; break; }
        if (nobodys) {
          unsigned char* row = v_smem + vs * V_BYTES + r * 128;
#pragma unroll
          for (int c = 0; c < 8; ++c) {              // (lanes start at different pieces: no bank conflicts)
            *reinterpret_cast<uint4*>(row + ((c ^ (r & 7)) << 4)) = make_uint4(0, 0, 0, 0);
            *reinterpret_cast<uint4*>(row + RT_PART_BYTES + ((c ^ (r & 7)) << 4)) = make_uint4(0, 0, 0, 0);
          }
          kvb_fence_async_shared();                  // generic writes -> visible to the product's reads
        }
        __syncwarp();
      }
      kvb_tc5_wait_st();
      kvb_tc5_fence_before();
      kvb_mbar_arrive(&p_ready[x]);
    }
    if (ok && n_mine > 0 && !RT_WAIT(&pv_done[x], (n_mine - 1) & 1)) ok = false;
    if (ok && n_mine > 0) {
      kvb_tc5_fence_after();
      if (p.sink != nullptr && row_sum > 0.0f) row_sum += exp2f(p.sink[hq] * 1.4426950408889634f - row_max);   // counts once
      const float inv = row_sum == 0.0f ? 0.0f : 1.0f / row_sum;     // a sink that is no number leaves none
      float o[4][32];
#pragma unroll
      for (int c = 0; c < 4; ++c) kvb_tc5_ld32(o_addr + c * 32, o[c]);
      kvb_tc5_wait_ld();
      if (row_valid) {
        const size_t at = (size_t)(q_begin + flat / p.G) * p.out_token + (size_t)hq * p.out_head + slice * RT_V;
        if (p.out_f32) {
          float* dst = (float*)p.out + at;
#pragma unroll
          for (int c = 0; c < 4; ++c)
#pragma unroll
            for (int i = 0; i < 32; i += 4)
              *reinterpret_cast<float4*>(dst + c * 32 + i) =
                  make_float4(o[c][i] * inv, o[c][i + 1] * inv, o[c][i + 2] * inv, o[c][i + 3] * inv);
        } else {
          bf16* dst = (bf16*)p.out + at;
#pragma unroll
          for (int c = 0; c < 4; ++c)
#pragma unroll
            for (int i = 0; i < 32; i += 8) {
              Vec16<bf16> packed;
#pragma unroll
              for (int n = 0; n < 8; ++n) packed.set(n, o[c][i + n] * inv);
              packed.store(dst + c * 32 + i);
            }
        }
      }
    } else if (!ok) {
      atomicOr(p.status, KVB_STATUS_WAIT_TIMEOUT);
      atomicExch(abort_flag, 1);
    }
  }

  // ---- everyone meets; the allocating warp frees the tensor memory ----
  kvb_tc5_fence_before();
  __syncthreads();
  if (warp == 10) {
    kvb_tc5_fence_after();
    kvb_tc5_dealloc(tmem_base, 512u);
  }
}

// ---- host side -----------------------------------------------------------------------------
// [rows, columns] of a plane with `pitch` elements a row, boxes of 64 columns of `box_rows` rows, 128-byte swizzle.
static bool rt_rows_map(CUtensorMap* map, const void* base, long long columns, long long rows, long long pitch, int box_rows) {
  KvbEncodeTiledFn encode = kvb_encode_tiled_fn();
  if (encode == nullptr) return false;
  const cuuint64_t dims[2] = {(cuuint64_t)columns, (cuuint64_t)rows};
  const cuuint64_t strides[1] = {(cuuint64_t)pitch * sizeof(bf16)};
  const cuuint32_t box[2] = {64, (cuuint32_t)box_rows};
  const cuuint32_t elem[2] = {1, 1};
  return encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, elem,
                CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int KH, bool SLOPE>
static cudaError_t launch_rows_tc5(dim3 grid, const CUtensorMap& k_map, const CUtensorMap& v_map, const CUtensorMap& q_map,
                                   const RowsTc5Params& p, cudaStream_t stream) {
  constexpr int smem = (4 * KH + (KH == 2 ? 4 : 2)) * RT_PART_BYTES + 16 * 8;
  static_assert(smem <= 227 * 1024, "the stages fit an SM");
  const cudaError_t err = cudaFuncSetAttribute(flash_rows_tc5_kernel<KH, SLOPE>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (err != cudaSuccess) return err;
  return kvb_launch((flash_rows_tc5_kernel<KH, SLOPE>), grid, dim3(RT_THREADS), smem, stream, true, k_map, v_map, q_map, p);
}

// keys, values: head 0 of slot 0 of page 0; `pitch` elements between two rows (a page's rows lie one behind the other, and
// so do the pages), `k_head` / `v_head` between two heads of a row.  `in_order`: pages of one row, and the rows of a
// request's visible positions are neighbours in ascending order.
extern "C" int kvb_flash_rows_tc5(void* out, long long out_token, long long out_head, int out_f32, const void* q,
                                  long long q_token, long long q_head, const void* keys, const void* values, long long pitch,
                                  int k_head, int v_head, const int* table, int table_stride, const int* query_start,
                                  const int* context_lens, const float* sink, const float* slopes, int num_reqs,
                                  int max_query_len, int num_tokens, int value_heads, int group, int maps, int DK, int DV,
                                  int page_size, int num_pages, float scale, int window, int in_order, cudaStream_t stream) {
  if (num_reqs == 0 || num_tokens == 0) return 0;
  KVB_REQUIRE(DK == 128 || DK == 192, "rows attention (tcgen05): keys of 128 or 192 entries");
  KVB_REQUIRE(DV > 0 && DV % RT_V == 0, "rows attention (tcgen05): values of a multiple of 128 entries");
  KVB_REQUIRE(in_order ? page_size == 1 : page_size == 8 || page_size == 16 || page_size == 32 || page_size == 64,
              "rows attention (tcgen05): pages of 8, 16, 32 or 64 rows, or rows in order");
  KVB_REQUIRE(value_heads > 0 && group > 0 && maps > 0 && num_reqs <= 65535, "rows attention (tcgen05): bad sizes");
  KVB_REQUIRE(aligned16(q) && aligned16(out) && aligned16(keys) && aligned16(values) && q_token % 8 == 0 && q_head % 8 == 0 &&
              pitch % 8 == 0 && k_head % 8 == 0 && v_head % 8 == 0 && out_token % (out_f32 ? 4 : 8) == 0 &&
              out_head % (out_f32 ? 4 : 8) == 0, "rows attention (tcgen05): rows must start on 16-byte boundaries");
  KVB_REQUIRE((long long)num_pages * page_size < (1ll << 31), "rows attention (tcgen05): too many rows");
  KVB_REQUIRE(scale > 0.0f, "rows attention (tcgen05): the scale must be positive");
  RowsTc5Params p = {};
  p.out = out; p.out_token = out_token; p.out_head = out_head; p.out_f32 = out_f32;
  p.q = (const bf16*)q; p.q_token = q_token; p.q_head = q_head;
  p.table = table; p.table_stride = table_stride; p.query_start = query_start; p.context_lens = context_lens;
  p.G = group; p.maps = maps; p.slices = DV / RT_V; p.page_rows = in_order ? RT_BN : page_size; p.num_pages = num_pages;
  p.window = window; p.in_order = in_order; p.k_head = k_head; p.v_head = v_head;
  p.scale_log2 = scale * 1.4426950408889634f;
  p.sink = sink; p.slopes = slopes; p.status = kvb_status_word();
  KVB_REQUIRE(p.status != nullptr, "rows attention (tcgen05): no status word");
  const long long rows = (long long)num_pages * page_size;
  p.no_row = (int)rows;
  alignas(64) CUtensorMap k_map, v_map, q_map;
  memset(&q_map, 0, sizeof(q_map));
  KVB_REQUIRE(rt_rows_map(&k_map, keys, (long long)(value_heads * maps - 1) * k_head + DK, rows, pitch, p.page_rows) &&
              rt_rows_map(&v_map, values, (long long)(value_heads - 1) * v_head + DV, rows, pitch, p.page_rows),
              "rows attention (tcgen05): no tensor map for the keys or the values");
  // the queries as [token][key head][head of the group][DK], as attention_prefill_tc5.cu has them (one map a value head);
  // strides that no tensor map describes (a row that serves all tokens has a stride of zero) leave them to be copied
  if (maps == 1 && RT_BM % group == 0 && q_token > 0 && q_head > 0) {
    KvbEncodeTiledFn encode = kvb_encode_tiled_fn();
    const cuuint64_t dims[4] = {(cuuint64_t)DK, (cuuint64_t)group, (cuuint64_t)value_heads, (cuuint64_t)num_tokens};
    const cuuint64_t strides[3] = {(cuuint64_t)q_head * sizeof(bf16), (cuuint64_t)group * q_head * sizeof(bf16),
                                   (cuuint64_t)q_token * sizeof(bf16)};
    const cuuint32_t box[4] = {64, (cuuint32_t)group, 1, (cuuint32_t)(RT_BM / group)};
    const cuuint32_t elem[4] = {1, 1, 1, 1};
    p.q_by_tma = encode(&q_map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(q), dims, strides, box, elem,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
  }
  const long long all_rows = (long long)max_query_len * group, heads = (long long)value_heads * maps * p.slices;
  p.tiles = kvb_tc5_query_tiles(heads * num_reqs * ((all_rows + 2 * RT_BM - 1) / (2 * RT_BM)));
  const long long pairs = (all_rows + p.tiles * RT_BM - 1) / (p.tiles * RT_BM);
  KVB_REQUIRE(pairs <= 65535, "rows attention (tcgen05): portion too long for one launch");
  const dim3 grid(value_heads * maps * p.slices, num_reqs, (unsigned)pairs);
  cudaError_t err;
  if (DK == 128) err = slopes ? launch_rows_tc5<2, true>(grid, k_map, v_map, q_map, p, stream) : launch_rows_tc5<2, false>(grid, k_map, v_map, q_map, p, stream);
  else err = slopes ? launch_rows_tc5<3, true>(grid, k_map, v_map, q_map, p, stream) : launch_rows_tc5<3, false>(grid, k_map, v_map, q_map, p, stream);
  KVB_CHECK_CUDA(err);
  KVB_CHECK_LAUNCH();
  return 0;
}

KVB_TRACE_TU(attention_rows_tc5)
