// Paged attention, general kernels: any head size up to 256, any head counts, any mix of
// prompt portions and decode tokens, optional sliding window (with an optional number of first
// positions that stay visible behind it), float or bf16 storage.  The attention of the 32-bit
// path; the bf16 path uses it for shapes its faster kernels refuse.
//
// A row is a (token, query head) pair.  What is computed for it depends on its position alone, never
// on how the step was cut or batched, so that a row has the same bits under any cutting:
//   * the cached positions fall into chunks of 64 (from position 0 on);
//   * a score is one accumulator in ascending d, times the scale; a chunk has its own maximum and sum of exponentials
//     (lanes hold keys n and n + 32, then a butterfly), and an output entry one accumulator over its keys in ascending order;
//   * chunks are added to the row's result one after the other (`Folded`); one without weight for the row is passed over.
// A key the row does not see has no part in any of it, whatever its value holds (a later token's may be no number): in
// chunks that not every row sees whole, an entry's sum passes over the keys that its row does not see.
//
// Two kernels do exactly that:
//   attention_tile: 32 or 64 rows of one request and kv head a block (portions of prompts).  Keys and values
//     of a chunk lie in shared memory and serve all rows, 4 x 4 scores and 4 x 4 NJ outputs a thread.
//     Bound by the shared-memory reads that feed the FMA units, or, for few blocks, by the longest of them.
//   attention_few: 8 rows a block, a warp a row.  At most 8 rows (decoded tokens): the chunks of a request go to
//     different blocks and a third kernel folds them; bound by the reading of keys and values.  A short portion of a
//     prompt within the first positions: its rows go to different blocks; bound by the latency of its few loads.
// Which one takes a request (att_request) follows its rows (new tokens times query heads a kv head): a tile
// costs all its rows' arithmetic however few there are.
// 32-bit, 24 heads of 128 over 8 kv heads (B200, call by call, cold caches; with segments of 256 positions walked by one block
// and tiles of 64 rows before): a portion of 250 tokens beside 6 decoded ones behind 750 to 1,000 cached 102 us (151 to 165);
// the portion alone 64 (86 to 94), the decoded ones 34 (66); one token behind 1,000, 16 heads over 4: 22 (60); 8 behind 8,192,
// 32 heads over 8: 182 (310); one behind 32,768, 16 heads over 4: 162 (198); 64 behind 200: 33 (51); a prompt of 2,048: 814
// (1,020).

// Cache layout: [pages, KVH, page_size, D]; page ids come from table[req, pos / page_size].
#include "common.cuh"

#define ATT_MAX_D 256
#define ATT_THREADS 256
#define ATT_CHUNK 64
#define ATT_FEW 8
#define ATT_FEW_TOKENS 32      // of a short portion: one lane each
#define ATT_ALONE 256          // positions up to which decoded tokens have one block a (request, kv head)
#define ATT_PORTION_END 256    // positions in front of which a short portion goes by eights of rows

template <typename T>
struct AttParams {
  T* out; const T* q; const T* k_cache; const T* v_cache;
  const int* table; const int* positions; const int* query_start;
  int out_stride, q_stride, table_stride, H, KVH, D, page_size, num_pages, window, keep_first, vec, chunks, reqs, part_rows;
  int parts;                 // blocks of attention_few a (request, kv head)
  int head0;                 // the first (request, kv head) of this launch of attention_few and of the fold behind it
  float scale;
  float* partial;            // [(request, kv head) of a launch, chunks, part_rows, D + 2]: accumulators, maximum, sum
  int* status;
};

// A row's result over the chunks so far: maximum M, sum L; each of its accumulators a becomes a_factor * a +
// s_factor * (the chunk's accumulator).
struct Folded {
  float M, L;
  float a_factor, s_factor;
  // l is not zero: the chunk holds a visible key.  (Where every score is NaN, m is still -INFINITY, l is NaN, and so
  // are the factors and the result.)
  __device__ __forceinline__ void fold(float m, float l) {
    const float top = fmaxf(M, m);
    a_factor = M == -INFINITY ? 0.0f : expf(M - top);
    s_factor = expf(m - top);
    L = fmaf(l, s_factor, __fmul_rn(L, a_factor));
    M = top;
  }
};

// One chunk's scores of a row, keys `lane` and `lane + 32` (-INFINITY: not seen), become probabilities, with their maximum
// and sum.
__device__ __forceinline__ void att_softmax(float& s0, float& s1, float& m, float& l) {
  m = warp_max(fmaxf(s0, s1));
  s0 = s0 == -INFINITY ? 0.0f : expf(s0 - m);
  s1 = s1 == -INFINITY ? 0.0f : expf(s1 - m);
  l = warp_sum(s0 + s1);
}

__device__ __forceinline__ float4 att_load4(const float* p, int valid, int vec) {
  if (vec) return *reinterpret_cast<const float4*>(p);
  return make_float4(p[0], valid > 1 ? p[1] : 0.0f, valid > 2 ? p[2] : 0.0f, valid > 3 ? p[3] : 0.0f);
}
__device__ __forceinline__ float4 att_load4(const bf16* p, int valid, int vec) {
  if (vec) {
    const uint2 raw = *reinterpret_cast<const uint2*>(p);
    return make_float4(__uint_as_float(raw.x << 16), __uint_as_float(raw.x & 0xffff0000u), __uint_as_float(raw.y << 16),
                       __uint_as_float(raw.y & 0xffff0000u));
  }
  return make_float4(to_float(p[0]), valid > 1 ? to_float(p[1]) : 0.0f, valid > 2 ? to_float(p[2]) : 0.0f,
                     valid > 3 ? to_float(p[3]) : 0.0f);
}

// Where some row of a block does not see a whole chunk, this stands for the probability of a key that its row does not see.
#define ATT_UNSEEN -1.0f

// A request's new tokens, rows a kv head and last position, and which kernel takes it.  By all threads of a warp.
// A portion of 3, 9, 16 and 32 tokens without cached ones, 24 heads of 128 over 8 (B200, call by call): 5.5, 5.6, 6.2 and
// 7.6 us by eights of rows, 15.4, 16.5, 17.6 and 18.8 in tiles; 64 tokens 22 in tiles.  16 tokens behind 100: 16 and 34.
struct AttRequest { int begin, rows, last; bool few, portion; };
template <typename T>
__device__ __forceinline__ AttRequest att_request(const AttParams<T>& p, int req) {
  const int begin = p.query_start[req], tokens = p.query_start[req + 1] - begin, lane = threadIdx.x & 31;
  AttRequest a = {begin, tokens * (p.H / p.KVH), 0, false, false};
  if (tokens <= ATT_FEW_TOKENS) {
    a.last = __reduce_max_sync(0xffffffffu, lane < tokens ? p.positions[begin + lane] : -1);
    a.few = a.rows <= ATT_FEW;
    a.portion = !a.few && a.last < ATT_PORTION_END;
  }
  return a;
}

__device__ __forceinline__ void att_copies_done() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

// What both kernels share: which keys the rows see, and the chunk in shared memory.
template <typename T>
struct AttBlock {
  const AttParams<T>& p;
  int req, kvh, G, begin, rows, row0;      // rows of this block: row0 .. row0 + rows - 1 of the request's
  int lo, hi, kept;                        // keys some row sees: [0, kept) and [lo, hi)
  int all_lo, all_hi;                      // keys every row sees: [all_lo, all_hi)
  long long head_off, page_elems;

  __device__ __forceinline__ int position(int r) const { return p.positions[begin + (row0 + r) / G]; }
  __device__ __forceinline__ int first_of(int pos) const { return p.window > 0 ? max(0, pos - p.window + 1) : 0; }
  // all threads; `pos` [rows] in shared memory is filled, barrier included
  __device__ __forceinline__ void look(int* pos, int* ends) {
    if (threadIdx.x == 0) { ends[0] = ends[4] = 0x7fffffff; ends[1] = ends[2] = ends[3] = 0; }
    __syncthreads();
    for (int r = threadIdx.x; r < rows; r += blockDim.x) {
      const int at = position(r), first = first_of(at);
      pos[r] = at;
      atomicMin(&ends[0], first);
      atomicMax(&ends[1], at + 1);
      atomicMax(&ends[2], min(p.keep_first, first));
      atomicMax(&ends[3], first);
      atomicMin(&ends[4], at + 1);
    }
    __syncthreads();
    lo = ends[0]; hi = ends[1]; kept = ends[2]; all_lo = ends[3]; all_hi = ends[4];
  }
  __device__ __forceinline__ bool ragged(int base) const { return base < all_lo || base + ATT_CHUNK > all_hi; }
  __device__ __forceinline__ bool wanted(int key) const { return (key >= lo && key < hi) || key < kept; }
  __device__ __forceinline__ bool chunk_wanted(int base) const {
    return (base + ATT_CHUNK > lo && base < hi) || base < kept;
  }
  __device__ __forceinline__ bool seen(int key, int pos) const {
    const int first = first_of(pos);
    return key <= pos && (key >= first || key < min(p.keep_first, first));
  }
  // Offset of a key in the cache (-1: nobody's, or a bad page, which is reported).
  __device__ __forceinline__ long long find(int key) const {
    if (!wanted(key)) return -1;
    const int page = p.table[(size_t)req * p.table_stride + key / p.page_size];
    if (page > 0 && page < p.num_pages) return (long long)page * page_elems + head_off + (long long)(key % p.page_size) * p.D;
    atomicOr(p.status, KVB_STATUS_BAD_PAGE);
    return -1;
  }
  // Keys of a chunk up to the last that somebody sees (what shared memory holds behind them counts for nothing).
  __device__ __forceinline__ int keys_of(int base) const { return min(ATT_CHUNK, max(hi, kept) - base); }
  // `keys` rows of a plane's chunk into shared memory as floats, `width` (a multiple of four) a row, zeros behind D; whole
  // pieces of 32-bit rows on their own (att_copies_done), lanes in powers of two sharing a key.
  template <int THREADS>
  __device__ __forceinline__ void fetch(float* dst, int stride, int width, const T* plane, const long long* offset, int keys) {
    const int pieces = width >> 2;
    if (sizeof(T) == 4 && p.vec) {
      const int log = pieces >= 32 ? 5 : 32 - __clz(pieces - 1);               // (one piece: __clz(0) is 32)
      for (int key = threadIdx.x >> log; key < keys; key += THREADS >> log) {
        const long long at = offset[key];
        for (int d = (threadIdx.x & ((1 << log) - 1)) << 2; d < width; d += 4 << log) {
          const bool there = at >= 0 && d < p.D;
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"((unsigned)__cvta_generic_to_shared(dst + key * stride + d)),
                       "l"(plane + (there ? at + d : 0)), "r"(there ? 16 : 0) : "memory");
        }
      }
      return;
    }
#pragma unroll 8
    for (int e = threadIdx.x; e < keys * pieces; e += THREADS) {
      const int key = e / pieces, d = (e - key * pieces) << 2;
      const long long at = offset[key];
      float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      if (at >= 0 && d < p.D) v = att_load4(plane + at + d, p.D - d, p.vec);
      *reinterpret_cast<float4*>(dst + key * stride + d) = v;
    }
  }
  __device__ __forceinline__ void fetch_queries(float* dst, int stride, int width) {
    const int pieces = width >> 2;
    for (int e = threadIdx.x; e < rows * pieces; e += blockDim.x) {
      const int r = e / pieces, d = (e - r * pieces) << 2, row = row0 + r;
      const T* src = p.q + (size_t)(begin + row / G) * p.q_stride + (size_t)(kvh * G + row % G) * p.D;
      float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      if (d < p.D) {                       // rows of q lie anywhere: entry by entry
        v.x = to_float(src[d]);
        if (d + 1 < p.D) v.y = to_float(src[d + 1]);
        if (d + 2 < p.D) v.z = to_float(src[d + 2]);
        if (d + 3 < p.D) v.w = to_float(src[d + 3]);
      }
      *reinterpret_cast<float4*>(dst + r * stride + d) = v;
    }
  }
  __device__ __forceinline__ T* out_row(int r) const {
    const int row = row0 + r;
    return p.out + (size_t)(begin + row / G) * p.out_stride + (size_t)(kvh * G + row % G) * p.D;
  }
};

template <typename T, int NJ, int ROWS>    // NJ: output columns in runs of 64; ROWS rows a block, four threads a row
__global__ void __launch_bounds__(4 * ROWS)
attention_tile_kernel(AttParams<T> p) {
  KVB_KERNEL_PROLOGUE(KVB_TAG_ATTN_ROWS);
  constexpr int THREADS = 4 * ROWS, LS = ROWS + 4, RS = ROWS / 4;    // a thread's score rows lie RS apart
  // blocks: (request, kv head) fastest, then the tiles, those with the most keys first
  const int heads = p.reqs * p.KVH, head = blockIdx.x % heads, req = head / p.KVH, kvh = head % p.KVH, G = p.H / p.KVH;
  const AttRequest a = att_request(p, req);
  const int begin = a.begin, all_rows = a.rows;
  const int row0 = (gridDim.x / heads - 1 - blockIdx.x / heads) * ROWS;
  if (a.few || a.portion || row0 >= all_rows) return;
  extern __shared__ __align__(16) float smem[];
  const int DK = (p.D + 3) & ~3, LK = DK + 4;
  constexpr int DV = 64 * NJ;
  float* const qs = smem;                                            // [ROWS][LK]
  float* const ks = qs + ROWS * LK;                                  // [ATT_CHUNK][LK]
  float* const vs = ks + ATT_CHUNK * LK;                             // [ATT_CHUNK][DV]
  float* const ss = vs + ATT_CHUNK * DV;                             // [ATT_CHUNK][LS]: scores, then probabilities
  __shared__ long long offset[ATT_CHUNK];
  __shared__ int pos[ROWS], ends[5], by_row;                         // by_row: some row has no weight for any key of the chunk
  __shared__ float old_factor[ROWS], new_factor[ROWS], row_sum[ROWS];
  AttBlock<T> b{p, req, kvh, G, begin, min(ROWS, all_rows - row0), row0, 0, 0, 0, 0, 0,
                (long long)kvh * p.page_size * p.D, (long long)p.KVH * p.page_size * p.D};
  b.look(pos, ends);
  b.fetch_queries(qs, LK, DK);
  // lanes of a warp: 4 x 8 threads, neighbours sharing a row, so that a warp's 16-byte reads are few distinct lines
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int ty = (warp >> 1) * 4 + (lane & 1) + 2 * (lane >> 4), tx = (warp & 1) * 8 + ((lane >> 1) & 7);
  float sum[4][4 * NJ];
  Folded total[8];                                                   // of the rows whose probabilities this warp forms
#pragma unroll
  for (int n = 0; n < 8; ++n) total[n] = Folded{-INFINITY, 0.0f, 0.0f, 0.0f};
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4 * NJ; ++j) sum[i][j] = 0.0f;

  for (int base = 0; base < b.hi; base += ATT_CHUNK) {
    if (!b.chunk_wanted(base)) continue;
    __syncthreads();                                                 // the chunk in front has been read
    if (threadIdx.x < ATT_CHUNK) offset[threadIdx.x] = b.find(base + threadIdx.x);
    if (threadIdx.x == 0) by_row = 0;
    __syncthreads();
    const int keys = b.keys_of(base);
    b.template fetch<THREADS>(ks, LK, DK, p.k_cache, offset, keys);
    b.template fetch<THREADS>(vs, DV, DV, p.v_cache, offset, keys);
    att_copies_done();
    __syncthreads();
    float s[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) s[i][j] = 0.0f;
#pragma unroll 2
    for (int d = 0; d < DK; d += 4) {
      float4 qv[4], kv[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) qv[i] = *reinterpret_cast<const float4*>(qs + (ty + RS * i) * LK + d);
#pragma unroll
      for (int j = 0; j < 4; ++j) kv[j] = *reinterpret_cast<const float4*>(ks + (tx + 16 * j) * LK + d);
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          s[i][j] = fmaf(kv[j].x, qv[i].x, s[i][j]);
          s[i][j] = fmaf(kv[j].y, qv[i].y, s[i][j]);
          s[i][j] = fmaf(kv[j].z, qv[i].z, s[i][j]);
          s[i][j] = fmaf(kv[j].w, qv[i].w, s[i][j]);
        }
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int key = tx + 16 * j;
      const bool there = offset[key] >= 0;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int r = ty + RS * i;
        ss[key * LS + r] = there && r < b.rows && b.seen(base + key, pos[r]) ? __fmul_rn(s[i][j], p.scale) : -INFINITY;
      }
    }
    __syncthreads();
    // all rows' softmaxes before any is folded, so that their shuffles overlap: 24 heads of 128 over 8 in bf16, 1,000 tokens, 431 us for
    // 452
    float m[8], l[8];
#pragma unroll
    for (int n = 0; n < 8; ++n) {
      const int r = warp * 8 + n;
      float s0 = ss[lane * LS + r], s1 = ss[(lane + 32) * LS + r];
      att_softmax(s0, s1, m[n], l[n]);
      ss[lane * LS + r] = s0;
      ss[(lane + 32) * LS + r] = s1;
    }
#pragma unroll
    for (int n = 0; n < 8; ++n) {
      const int r = warp * 8 + n;
      // a row for which the chunk has no weight (none of it seen, or every score -infinity) keeps what it has
      if (l[n] != 0.0f) {
        total[n].fold(m[n], l[n]);
      } else if (r < b.rows) {
        ss[lane * LS + r] = ss[(lane + 32) * LS + r] = ATT_UNSEEN;
        if (lane == 0) by_row = 1;
      }
      if (lane == 0) { old_factor[r] = l[n] != 0.0f ? total[n].a_factor : 1.0f; new_factor[r] = l[n] != 0.0f ? total[n].s_factor : 0.0f; }
    }
    __syncwarp();
    const bool ragged = b.ragged(base);
    if (ragged)
      for (int n = 0; n < 8; ++n) {
        const int r = warp * 8 + n;
        if (!b.seen(base + lane, pos[r])) ss[lane * LS + r] = ATT_UNSEEN;
        if (!b.seen(base + lane + 32, pos[r])) ss[(lane + 32) * LS + r] = ATT_UNSEEN;
      }
    __syncthreads();
    float acc[4][4 * NJ];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4 * NJ; ++j) acc[i][j] = 0.0f;
    auto add_key = [&](int key, bool some) {                         // `some`: only to the rows that see the key
      const float4 pr = *reinterpret_cast<const float4*>(ss + key * LS + ty * 4);
#pragma unroll
      for (int j = 0; j < NJ; ++j) {
        const float4 v = *reinterpret_cast<const float4*>(vs + key * DV + j * 64 + tx * 4);
        const float w[4] = {pr.x, pr.y, pr.z, pr.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          if (some && w[i] == ATT_UNSEEN) continue;
          acc[i][4 * j] = fmaf(w[i], v.x, acc[i][4 * j]);
          acc[i][4 * j + 1] = fmaf(w[i], v.y, acc[i][4 * j + 1]);
          acc[i][4 * j + 2] = fmaf(w[i], v.z, acc[i][4 * j + 2]);
          acc[i][4 * j + 3] = fmaf(w[i], v.w, acc[i][4 * j + 3]);
        }
      }
    };
    if (ragged || by_row) {
#pragma unroll 4
      for (int key = 0; key < keys; ++key) add_key(key, true);
    } else {
#pragma unroll 4
      for (int key = 0; key < ATT_CHUNK; ++key) add_key(key, false);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float was = old_factor[ty * 4 + i], is = new_factor[ty * 4 + i];
#pragma unroll
      for (int j = 0; j < 4 * NJ; ++j) sum[i][j] = fmaf(acc[i][j], is, __fmul_rn(sum[i][j], was));
    }
  }
  if (lane == 0)
#pragma unroll
    for (int n = 0; n < 8; ++n) row_sum[warp * 8 + n] = total[n].L;
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int r = ty * 4 + i;
    if (r >= b.rows) continue;
    const float L = row_sum[r], inv = L > 0.0f ? 1.0f / L : 0.0f;
    T* to = b.out_row(r);
#pragma unroll
    for (int j = 0; j < NJ; ++j)
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const int d = j * 64 + tx * 4 + c;
        if (d < p.D) to[d] = from_float<T>(sum[i][4 * j + c] * inv);
      }
  }
}

template <typename T, int NJ>              // NJ: output columns in runs of 64
__global__ void __launch_bounds__(ATT_THREADS, NJ == 1 ? 4 : 3)
attention_few_kernel(AttParams<T> p) {
  KVB_KERNEL_PROLOGUE(KVB_TAG_ATTN_ROWS);
  // blocks: the chunks of a (request, kv head) dealt out in turn, or its rows eight by eight, next to one another
  const int head = p.head0 + blockIdx.x / p.parts, part_no = blockIdx.x % p.parts;
  const int req = head / p.KVH, kvh = head % p.KVH, G = p.H / p.KVH;
  const AttRequest a = att_request(p, req);
  const int row0 = a.few ? 0 : part_no * ATT_FEW, begin = a.begin;
  if (!(a.few || a.portion) || row0 >= a.rows) return;
  // chunks of a decoded token: every parts-th (the fold does not read what was not written), as many as scratch is bound to hold
  const bool apart = a.few && p.chunks > 1;                          // the fold adds the chunks up
  const int first_chunk = apart ? part_no : 0, step = apart ? p.parts : 1;
  const int end_chunk = apart ? min(a.last / ATT_CHUNK + 1, p.chunks) : a.last / ATT_CHUNK + 1;
  if (first_chunk >= end_chunk || (a.few && !apart && part_no > 0)) return;
  const int r = threadIdx.x >> 5, lane = threadIdx.x & 31, rows = min(ATT_FEW, a.rows - row0);     // a warp a row
  const bool live = r < rows;
  // every warp looks the rows up for itself, a lane a row
  const int at = lane < rows ? p.positions[begin + (row0 + lane) / G] : -1, mine = __shfl_sync(0xffffffffu, at, live ? r : 0);
  extern __shared__ __align__(16) float smem[];
  const int DK = (p.D + 3) & ~3, LK = DK + 4;
  constexpr int DV = 64 * NJ, RUNS = (NJ + 1) / 2;                   // a lane's quads of output columns: 128 apart
  float* const qs = smem;                                            // [ATT_FEW][LK]
  float* const ks = qs + ATT_FEW * LK;                               // [ATT_CHUNK][LK]
  float* const vs = ks + ATT_CHUNK * LK;                             // [ATT_CHUNK][DV]
  __shared__ long long offset[ATT_CHUNK];
  __shared__ float probability[ATT_FEW][ATT_CHUNK];
  AttBlock<T> b{p, req, kvh, G, begin, rows, row0, 0, 0, 0, 0, 0,
                (long long)kvh * p.page_size * p.D, (long long)p.KVH * p.page_size * p.D};
  {
    const int first = b.first_of(at);
    b.lo = __reduce_min_sync(0xffffffffu, at < 0 ? 0x7fffffff : first);
    b.hi = __reduce_max_sync(0xffffffffu, at) + 1;
    b.kept = __reduce_max_sync(0xffffffffu, at < 0 ? 0 : min(p.keep_first, first));
    b.all_lo = b.first_of(mine);           // all the rows of a warp: one
    b.all_hi = mine + 1;
  }
  bool any = false;
  float sum[RUNS][4];                      // a portion's rows over their chunks
  Folded total{-INFINITY, 0.0f, 0.0f, 0.0f};
#pragma unroll
  for (int j = 0; j < RUNS; ++j) sum[j][0] = sum[j][1] = sum[j][2] = sum[j][3] = 0.0f;
  for (int chunk = first_chunk; chunk < end_chunk; chunk += step) {
    const int base = chunk * ATT_CHUNK;
    float* const part = p.partial + (((size_t)(blockIdx.x / p.parts) * p.chunks + chunk) * p.part_rows + r) * (p.D + 2);
    if (!b.chunk_wanted(base)) {
      if (apart && live && lane == 0) part[p.D + 1] = 0.0f;
      continue;
    }
    const long long found = threadIdx.x < ATT_CHUNK ? b.find(base + threadIdx.x) : -1;
    if (any) __syncthreads();                                        // the chunk in front has been read
    else b.fetch_queries(qs, LK, DK);
    any = true;
    if (threadIdx.x < ATT_CHUNK) offset[threadIdx.x] = found;
    __syncthreads();
    const int keys = b.keys_of(base);
    b.template fetch<ATT_THREADS>(ks, LK, DK, p.k_cache, offset, keys);
    b.template fetch<ATT_THREADS>(vs, DV, DV, p.v_cache, offset, keys);
    att_copies_done();
    __syncthreads();
    if (!live) continue;
    float s0 = 0.0f, s1 = 0.0f;
#pragma unroll 4
    for (int d = 0; d < DK; d += 4) {
      const float4 q = *reinterpret_cast<const float4*>(qs + r * LK + d);
      const float4 a = *reinterpret_cast<const float4*>(ks + lane * LK + d);
      const float4 c = *reinterpret_cast<const float4*>(ks + (lane + 32) * LK + d);
      s0 = fmaf(a.x, q.x, s0); s0 = fmaf(a.y, q.y, s0); s0 = fmaf(a.z, q.z, s0); s0 = fmaf(a.w, q.w, s0);
      s1 = fmaf(c.x, q.x, s1); s1 = fmaf(c.y, q.y, s1); s1 = fmaf(c.z, q.z, s1); s1 = fmaf(c.w, q.w, s1);
    }
    const bool sees0 = b.seen(base + lane, mine), sees1 = b.seen(base + lane + 32, mine);
    s0 = offset[lane] >= 0 && sees0 ? __fmul_rn(s0, p.scale) : -INFINITY;
    s1 = offset[lane + 32] >= 0 && sees1 ? __fmul_rn(s1, p.scale) : -INFINITY;
    float m, l;
    att_softmax(s0, s1, m, l);
    if (!sees0) s0 = ATT_UNSEEN;
    if (!sees1) s1 = ATT_UNSEEN;
    probability[r][lane] = s0;
    probability[r][lane + 32] = s1;
    __syncwarp();
    float acc[RUNS][4];
#pragma unroll
    for (int j = 0; j < RUNS; ++j) acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0.0f;
    auto add_key = [&](int key, bool some) {                         // `some`: not if the row does not see the key
      const float w = probability[r][key];
      if (some && w == ATT_UNSEEN) return;
#pragma unroll
      for (int j = 0; j < RUNS; ++j) {
        const int d = j * 128 + lane * 4;
        if (d < DV) {
          const float4 v = *reinterpret_cast<const float4*>(vs + key * DV + d);
          acc[j][0] = fmaf(w, v.x, acc[j][0]);
          acc[j][1] = fmaf(w, v.y, acc[j][1]);
          acc[j][2] = fmaf(w, v.z, acc[j][2]);
          acc[j][3] = fmaf(w, v.w, acc[j][3]);
        }
      }
    };
    if (b.ragged(base)) {
      for (int key = 0; key < keys; ++key) add_key(key, true);
    } else {
#pragma unroll 8
      for (int key = 0; key < ATT_CHUNK; ++key) add_key(key, false);
    }
    __syncwarp();                                                    // the probabilities have been read
    if (apart) {
#pragma unroll
      for (int j = 0; j < RUNS; ++j)
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const int d = j * 128 + lane * 4 + c;
          if (d < p.D && l != 0.0f) part[d] = acc[j][c];
        }
      if (lane == 0) { part[p.D] = m; part[p.D + 1] = l; }
    } else if (l != 0.0f) {
      total.fold(m, l);
#pragma unroll
      for (int j = 0; j < RUNS; ++j)
#pragma unroll
        for (int c = 0; c < 4; ++c) sum[j][c] = fmaf(acc[j][c], total.s_factor, __fmul_rn(sum[j][c], total.a_factor));
    }
  }
  if (!live || apart) return;
  const float inv = total.L > 0.0f ? 1.0f / total.L : 0.0f;
  T* to = b.out_row(r);
#pragma unroll
  for (int j = 0; j < RUNS; ++j)
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const int d = j * 128 + lane * 4 + c;
      if (d < p.D) to[d] = from_float<T>(sum[j][c] * inv);
    }
}

// Folds the chunks of the requests that attention_few took: a block a (request, kv head), a warp a row.  The next ATT_AHEAD
// chunks are on their way while these go one after the other.
#define ATT_AHEAD 8
template <typename T, int NJ>
__global__ void __launch_bounds__(ATT_THREADS)
attention_fold_kernel(AttParams<T> p) {
  KVB_KERNEL_PROLOGUE(KVB_TAG_ATTN_ROWS);
  const int head = p.head0 + blockIdx.x, req = head / p.KVH, kvh = head % p.KVH, G = p.H / p.KVH;
  const int begin = p.query_start[req], all_rows = (p.query_start[req + 1] - begin) * G;
  const int r = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (all_rows > ATT_FEW || r >= all_rows) return;
  constexpr int MOST = 2 * NJ;
  float sum[MOST];
#pragma unroll
  for (int j = 0; j < MOST; ++j) sum[j] = 0.0f;
  Folded total{-INFINITY, 0.0f, 0.0f, 0.0f};
  const int last = min(p.chunks - 1, p.positions[begin + r / G] / ATT_CHUNK);
  const size_t chunk_floats = (size_t)p.part_rows * (p.D + 2);
  const float* const parts = p.partial + ((size_t)blockIdx.x * p.chunks * p.part_rows + r) * (p.D + 2);
  struct Lot { float m[ATT_AHEAD], l[ATT_AHEAD], v[ATT_AHEAD][MOST]; };
  auto ask = [&](Lot& lot, int c0) {
#pragma unroll
    for (int n = 0; n < ATT_AHEAD; ++n) {
      const float* from = parts + (c0 + n) * chunk_floats;
      lot.l[n] = c0 + n <= last ? from[p.D + 1] : 0.0f;
      if (c0 + n > last) continue;
      lot.m[n] = from[p.D];                                          // (of a chunk without a visible key: not used)
#pragma unroll
      for (int j = 0; j < MOST; ++j)
        if (lane + 32 * j < p.D) lot.v[n][j] = from[lane + 32 * j];
    }
  };
  auto add = [&](const Lot& lot) {
#pragma unroll
    for (int n = 0; n < ATT_AHEAD; ++n) {
      if (lot.l[n] == 0.0f) continue;
      total.fold(lot.m[n], lot.l[n]);
#pragma unroll
      for (int j = 0; j < MOST; ++j)
        if (lane + 32 * j < p.D) sum[j] = fmaf(lot.v[n][j], total.s_factor, __fmul_rn(sum[j], total.a_factor));
    }
  };
  Lot here, next;
  ask(here, 0);
  for (int c0 = 0; c0 <= last; c0 += 2 * ATT_AHEAD) {
    ask(next, c0 + ATT_AHEAD);
    add(here);
    ask(here, c0 + 2 * ATT_AHEAD);
    add(next);
  }
  const float inv = total.L > 0.0f ? 1.0f / total.L : 0.0f;
  T* to = p.out + (size_t)(begin + r / G) * p.out_stride + (size_t)(kvh * G + r % G) * p.D;
#pragma unroll
  for (int j = 0; j < MOST; ++j)
    if (lane + 32 * j < p.D) to[lane + 32 * j] = from_float<T>(sum[j] * inv);
}

// What a batch launches, from its shape and a bound on its positions.
struct AttPlan {
  bool tile, few, fold;
  int chunks, part_rows, parts;        // of attention_few: see AttParams
  long long lot;                       // (request, kv head) pairs a launch of attention_few takes
  long long scratch;                   // floats
};
// One long context beside many short ones asks for as much as if all were long: pairs are taken in lots for which this
// many floats are enough (their blocks fill the GPU many times over by then).
#define ATT_SCRATCH_FLOATS (16 << 20)
static AttPlan att_plan(int reqs, int H, int KVH, int D, int max_query_len, int tokens, int bound) {
  AttPlan a = {false, false, false, 1, 1, 1, 1, 0};
  if (reqs <= 0 || KVH <= 0 || H < KVH || D <= 0 || max_query_len <= 0) return a;      // nothing to do, or refused below
  const long long G = H / KVH, most = max_query_len * G;
  const bool equal = (long long)max_query_len * reqs == tokens;      // only one kind of request
  const bool eight = G <= ATT_FEW && (most <= ATT_FEW || !equal);    // some may have at most 8 rows
  const bool portions = most > ATT_FEW && (max_query_len <= ATT_FEW_TOKENS || !equal);
  // up to ATT_ALONE positions a block walks all chunks itself: no scratch, no fold
  const int all = bound > ATT_ALONE ? (bound + ATT_CHUNK - 1) / ATT_CHUNK : 1;
  a.tile = most > ATT_FEW && (max_query_len > ATT_FEW_TOKENS || bound > ATT_PORTION_END);
  a.few = eight || portions;
  a.chunks = eight ? all : 1;
  a.fold = a.chunks > 1;
  a.part_rows = (int)(most < ATT_FEW ? most : ATT_FEW);
  // blocks a (request, kv head): one a chunk, but no more in all than eight times those that the GPU holds (a bound on the
  // positions is often far above them, and every block costs its start)
  const long long heads = (long long)reqs * KVH, sms = kvb_sm_count() > 0 ? kvb_sm_count() : 148, room = 24 * sms / heads + 1;
  a.parts = a.chunks < room ? a.chunks : (int)room;
  const long long groups = ((max_query_len < ATT_FEW_TOKENS ? max_query_len : ATT_FEW_TOKENS) * G + ATT_FEW - 1) / ATT_FEW;
  if (portions && groups > a.parts) a.parts = (int)groups;
  const long long each = (long long)a.chunks * a.part_rows * (D + 2);
  const long long fit = ATT_SCRATCH_FLOATS / each;
  a.lot = !a.fold || heads <= fit ? heads : fit < 1 ? 1 : fit;
  a.scratch = a.fold ? a.lot * each : 0;
  return a;
}

template <typename T, int NJ>
static int launch_attention(AttParams<T> p, const AttPlan& plan, int max_query_len, cudaStream_t stream) {
  constexpr int DV = 64 * NJ, MOST_LK = DV + 4;            // (what is allowed is the most that any D asks for: another
  const int LK = ((p.D + 3) & ~3) + 4;                     // thread's launch may lie between the allowance and this one's)
  auto tile_bytes = [](int lk, int rows) { return (int)sizeof(float) * (rows * lk + ATT_CHUNK * (lk + DV + rows + 4)); };
  auto few_bytes = [](int lk) { return (int)sizeof(float) * (ATT_FEW * lk + ATT_CHUNK * (lk + DV)); };
  const long long heads = (long long)p.reqs * p.KVH, most = (long long)max_query_len * (p.H / p.KVH);
  if (plan.tile) {
#define KVB_ATT_TILE(ROWS_)                                                                                                   \
    KVB_CHECK_CUDA(cudaFuncSetAttribute(attention_tile_kernel<T, NJ, ROWS_>, cudaFuncAttributeMaxDynamicSharedMemorySize,     \
                                        tile_bytes(MOST_LK, ROWS_)));                                                         \
    KVB_CHECK_CUDA(kvb_launch((attention_tile_kernel<T, NJ, ROWS_>), dim3((unsigned)(heads * ((most + ROWS_ - 1) / ROWS_))),  \
                              dim3(4 * ROWS_), tile_bytes(LK, ROWS_), stream, true, p))
    // Blocks of 64 rows that do not fill the GPU twice take as long as the longest of them: half of them is done sooner.
    // 24 heads of 128 over 8: 250 tokens 64 us for 86; 3 portions of 100 behind 700: 202 for 256.  Where keys and values do not go
    // on their own (bf16, rows off 16 bytes) half the threads take longer to bring a chunk: 6 heads of 40 over 2 in bf16, 4 portions
    // of 3 behind 4,000: 64 rows 720 us, 32 rows 820.
    const long long sms = kvb_sm_count() > 0 ? kvb_sm_count() : 148;
    if (sizeof(T) == 4 && p.vec && heads * ((most + 63) / 64) <= 2 * sms) { KVB_ATT_TILE(32); } else { KVB_ATT_TILE(64); }
#undef KVB_ATT_TILE
  }
  if (plan.few) {
    KVB_CHECK_CUDA(cudaFuncSetAttribute(attention_few_kernel<T, NJ>, cudaFuncAttributeMaxDynamicSharedMemorySize, few_bytes(MOST_LK)));
    for (long long head0 = 0; head0 < heads; head0 += plan.lot) {    // one behind the other: the scratch is the same
      const unsigned here = (unsigned)(heads - head0 < plan.lot ? heads - head0 : plan.lot);
      p.head0 = (int)head0;
      KVB_CHECK_CUDA(kvb_launch((attention_few_kernel<T, NJ>), dim3(here * p.parts), dim3(ATT_THREADS), few_bytes(LK), stream, true, p));
      if (plan.fold)
        KVB_CHECK_CUDA(kvb_launch((attention_fold_kernel<T, NJ>), dim3(here), dim3(ATT_THREADS), 0, stream, true, p));
    }
  }
  KVB_CHECK_LAUNCH();
  return 0;
}

template <typename T>
static int attention_of(const AttParams<T>& p, const AttPlan& plan, int max_query_len, cudaStream_t stream) {
  if (p.D <= 64) return launch_attention<T, 1>(p, plan, max_query_len, stream);
  if (p.D <= 128) return launch_attention<T, 2>(p, plan, max_query_len, stream);
  return launch_attention<T, 4>(p, plan, max_query_len, stream);
}

// Floats of the scratch, and the kernels that are launched.  `bound`: no request has more positions, cached and new.
extern "C" long long kvb_paged_attention_scratch(int num_reqs, int H, int KVH, int D, int max_query_len, int tokens, int bound) {
  return att_plan(num_reqs, H, KVH, D, max_query_len, tokens, bound).scratch;
}
extern "C" int kvb_paged_attention_launches(int num_reqs, int H, int KVH, int D, int max_query_len, int tokens, int bound) {
  const AttPlan a = att_plan(num_reqs, H, KVH, D, max_query_len, tokens, bound);
  const long long heads = (long long)num_reqs * KVH;
  return (a.tile ? 1 : 0) + (a.few ? (int)((heads + a.lot - 1) / a.lot) * (a.fold ? 2 : 1) : 0);
}

extern "C" int kvb_paged_attention_rows(void* out, int out_stride, const void* q, int q_stride,
                                        const void* k_cache, const void* v_cache, const int* table,
                                        int table_stride, const int* positions, const int* query_start, int num_reqs,
                                        int max_query_len, int tokens, int H, int KVH, int D, int page_size,
                                        int num_pages, float scale, int window, int keep_first, int bound, float* partial,
                                        int dtype, cudaStream_t stream) {
  if (tokens == 0 || num_reqs == 0) return 0;
  KVB_REQUIRE(D > 0 && D <= ATT_MAX_D, "paged_attention: head_dim must be in [1, 256]");
  KVB_REQUIRE(H > 0 && KVH > 0 && H % KVH == 0, "paged_attention: H must be a multiple of KVH");
  KVB_REQUIRE(page_size > 0 && num_pages > 1, "paged_attention: empty cache");
  KVB_REQUIRE(keep_first >= 0 && (keep_first == 0 || window > 0), "paged_attention: kept first positions need a window");
  KVB_REQUIRE((long long)tokens * H < (1ll << 31) && max_query_len > 0 && max_query_len <= tokens, "paged_attention: too many rows");
  const AttPlan plan = att_plan(num_reqs, H, KVH, D, max_query_len, tokens, bound);
  KVB_REQUIRE((long long)num_reqs * KVH * (((long long)max_query_len * (H / KVH) + 31) / 32) < (1ll << 31) &&
              plan.lot * plan.parts < (1ll << 31), "paged_attention: too many blocks for one launch");
  KVB_REQUIRE(plan.scratch == 0 || partial != nullptr, "paged_attention: no scratch");
  int* status = kvb_status_word();
  KVB_REQUIRE(status != nullptr, "paged_attention: no status word");
  const int esize = dtype == KVB_F32 ? 4 : 2;
  const int vec = D % 4 == 0 && ((uintptr_t)k_cache | (uintptr_t)v_cache) % (4 * esize) == 0;
#define KVB_ATT(T_)                                                                                                    \
  attention_of<T_>(AttParams<T_>{(T_*)out, (const T_*)q, (const T_*)k_cache, (const T_*)v_cache, table, positions,     \
                                 query_start, out_stride, q_stride, table_stride, H, KVH, D, page_size, num_pages,     \
                                 window, keep_first, vec, plan.chunks, num_reqs, plan.part_rows, plan.parts, 0,      \
                                 scale, partial, status},                                                              \
                   plan, max_query_len, stream)
  return dtype == KVB_F32 ? KVB_ATT(float) : KVB_ATT(bf16);
#undef KVB_ATT
}

KVB_TRACE_TU(attention_generic)
