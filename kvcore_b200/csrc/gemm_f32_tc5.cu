// 32-bit linear layer on the 5th-generation tensor cores without giving up 32-bit operands:
// out[m, n] = sum_k x[m, k] * w[n, k] (+ bias[n]), float in and out.
//
// A float is three bf16 numbers, exactly: the number rounded to bf16, what that left, times 2^8, rounded to bf16, and the rest, times
// 2^16 (8 + 8 + 8 bits; the factors keep the smallest float, 2^-149, above the smallest bf16, 2^-133.  In the pipe a number below
// 2^-126 stands as high as 2^-126: sums of such numbers only are off by up to half of 2^-149 of one a term).  Six of the nine products
// of such pieces are taken (bf16 x bf16 is exact in 32 bits); the three left out are below 2^-25, 2^-25 and 2^-34 of the
// product they belong to.  What limits the result is then how sums are taken.  The tensor pipe adds into its accumulator without
// rounding to nearest, so an accumulator holds 64 k only, small products first, and is then added to the sum proper in a
// register, rounded to nearest.  Error against 64 bits relative to the result, random inputs: 1.1e-7 to 1.5e-7 at K 2048 to
// 8192 where one accumulator in ascending k (gemm_f32.cu) has 8.1e-7 to 1.6e-6.  Sums of up to about 16 terms that are not zero
// are further off than there, by a unit in the last place: largest error in 2^-24 of the terms, this kernel and that one, one
// term 2.3 and 1.0, four 3.8 and 2.9, eight 3.2 and 4.0, 64 1.8 and 6.1, 2048 0.4 and 5.4.
//
// The order of the sums depends on N and K only: 64 k at a time in ascending order, within `segments` equal stretches of K
// (they give the SMs work where N has few tiles) whose sums are added in order.  Every number of rows takes this kernel
// (rows are columns of the tensor pipe's tile, 16 to 128 of them), so a row's bits do not depend on the batch.
//
// A block owns 128 columns of the layer (128 lanes of tensor memory), up to 128 rows and one stretch of K:
//   * one warp brings the weights as they are, by TMA, [128 columns] x [64 k] floats a chunk, the first of them before the
//     kernel in front has finished (weights are written by no kernel of a step);
//   * eight warps cut them to pieces (a thread owns a column and half of the chunk's k) and lay these in tensor memory,
//     where the product takes its A operand from: 48 KB that shared memory need not deliver twice;
//   * one warp brings the rows' pieces, cut once by a small kernel in front, by TMA;
//   * one warp issues the 24 products of a chunk; two accumulators of 128 columns alternate, and eight warps add the finished
//     one to their sums while the other fills.
// What bounds it: with 128 rows a block the tensor pipe (1,560 cycles a chunk, 1,536 of them products); with few the cutting
// (700 cycles a chunk of a warp's instructions, 1,420 with its waits).  Microseconds, cutting and adding of stretches
// included, this kernel and gemm_f32.cu: 256 rows, N 16384, K 3072 122 and 620 (210 and 42 TFLOP/s), N 5120, K 3072 60 and
// 283, N 3072, K 8192 77 and 424; 32 rows, N 16384, K 3072 54 and 174; 4 rows 52 and 74.
//
// Where the result is not finite the output is taken again in plain FMA (infinities would otherwise meet the zeros among
// the pieces and numbers above 3.39e38 would round to one): such outputs are as gemm_f32.cu has them, and cost a multiple of the
// finite ones (fs_by_fma).
#include <cuda.h>

#include "common.cuh"
#include "sm100.cuh"

#define FS_COLS 128                        // columns (weight rows) of a block
#define FS_K 64                            // k of a chunk
#define FS_W_BYTES (FS_COLS * FS_K * 4)
#define FS_TMEM_W 256                      // first column of the weights' pieces: two stages of 96 behind two accumulators of 128
#define FS_SPIN_LIMIT (1u << 20)
#define FS_MAX_PARTIAL_FLOATS (32ll << 20) // sums of stretches that wait in scratch: rows are taken in lots beyond that

struct SplitParams {
  float* out; long long ldo;               // where a block's sums go: the result, or [segments][rows][N] of scratch
  const float* bias;                       // with the result only
  const float* x; long long ldx; const float* w; int x16;   // for outputs that are not finite (x16: rows of x on 16-byte boundaries)
  int M, N, K;
  int tiles_m, tiles_n, segments, seg_chunks, chunks;
  int* status;
};

// Two floats at once, each rounded as a scalar instruction rounds it.
__device__ __forceinline__ float2 fs_fma2(float2 a, float b, float2 c) {
  float2 d;
  asm("{\n.reg .b64 x, y, z;\nmov.b64 x, {%2, %3};\nmov.b64 y, {%4, %4};\nmov.b64 z, {%5, %6};\n"
      "fma.rn.f32x2 x, x, y, z;\nmov.b64 {%0, %1}, x;\n}\n"
      : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b), "f"(c.x), "f"(c.y));
  return d;
}
__device__ __forceinline__ float2 fs_times2(float2 a, float b) {
  float2 d;
  asm("{\n.reg .b64 x, y;\nmov.b64 x, {%2, %3};\nmov.b64 y, {%4, %4};\nmul.rn.f32x2 x, x, y;\nmov.b64 {%0, %1}, x;\n}\n"
      : "=f"(d.x), "=f"(d.y) : "f"(a.x), "f"(a.y), "f"(b));
  return d;
}
// Two floats as three pairs of bf16 (the lower one in the lower half), exactly: hi + mid / 2^8 + lo / 2^16.
__device__ __forceinline__ void fs_cut(float a, float b, unsigned& hi, unsigned& mid, unsigned& lo) {
  float2 v = make_float2(a, b);
  __nv_bfloat162 h = __float22bfloat162_rn(v);
  hi = *reinterpret_cast<unsigned*>(&h);
  v = fs_times2(fs_fma2(make_float2(__uint_as_float(hi << 16), __uint_as_float(hi & 0xffff0000u)), -1.0f, v), 256.0f);
  __nv_bfloat162 m = __float22bfloat162_rn(v);
  mid = *reinterpret_cast<unsigned*>(&m);
  v = fs_times2(fs_fma2(make_float2(__uint_as_float(mid << 16), __uint_as_float(mid & 0xffff0000u)), -1.0f, v), 256.0f);
  __nv_bfloat162 l = __float22bfloat162_rn(v);
  lo = *reinterpret_cast<unsigned*>(&l);
}

// Outputs that are not finite, again, FS_AGAIN at a time that share a row (of x or of w): one accumulator each in ascending k, as
// gemm_f32.cu takes it.  Bound by the latency of the loads, eight k at a time.  Whole products of which some is infinite, now, with
// one output after the other four bytes at a time, and by gemm_f32.cu, microseconds: 256 rows, N 5120, K 3072: a row of x 511,
// 1,850, 289; a column of weights (every output) 6,250, 27,300, 288; N 16384: a row of weights 3,030, 13,300, 623; a column
// 8,500, 81,600, 624; finite 124.
#define FS_AGAIN 4
#define FS_AGAIN_QUADS 2
__device__ __forceinline__ float4 fs_load4(const float* p, bool vec) {
  return vec ? *reinterpret_cast<const float4*>(p) : make_float4(p[0], p[1], p[2], p[3]);
}
__device__ __noinline__ void fs_by_fma(float (&out)[FS_AGAIN], const float* one, bool one16, const float* const (&others)[FS_AGAIN],
                                       bool others16, int K) {
  float acc[FS_AGAIN];
  const float* row[FS_AGAIN];
#pragma unroll
  for (int r = 0; r < FS_AGAIN; ++r) { acc[r] = 0.0f; row[r] = others[r]; }
  bool any = true;
  for (int k = 0; k < K && any; k += 4 * FS_AGAIN_QUADS) {         // K is a multiple of four
    float4 a[FS_AGAIN_QUADS], b[FS_AGAIN_QUADS][FS_AGAIN];
#pragma unroll
    for (int i = 0; i < FS_AGAIN_QUADS; ++i) {
      const int at = min(k + 4 * i, K - 4);
      a[i] = fs_load4(one + at, one16);
#pragma unroll
      for (int r = 0; r < FS_AGAIN; ++r) b[i][r] = fs_load4(row[r] + at, others16);
    }
#pragma unroll
    for (int i = 0; i < FS_AGAIN_QUADS; ++i)
      if (k + 4 * i < K)
#pragma unroll
        for (int r = 0; r < FS_AGAIN; ++r) {
          acc[r] = fmaf(b[i][r].x, a[i].x, acc[r]);
          acc[r] = fmaf(b[i][r].y, a[i].y, acc[r]);
          acc[r] = fmaf(b[i][r].z, a[i].z, acc[r]);
          acc[r] = fmaf(b[i][r].w, a[i].w, acc[r]);
        }
    any = false;                                                   // a NaN stays one
#pragma unroll
    for (int r = 0; r < FS_AGAIN; ++r) any |= acc[r] == acc[r];
  }
#pragma unroll
  for (int r = 0; r < FS_AGAIN; ++r) out[r] = acc[r];
}

// x [M, K] -> pieces [3][M][Kp] bf16.  Four neighbouring k a thread (K is a multiple of four).
__global__ void __launch_bounds__(256) f32_pieces_kernel(bf16* pieces, const float* x, int M, int K, int Kp, long long ldx, int vec) {
  KVB_KERNEL_PROLOGUE(KVB_TAG_GEMM_F32);
  const int quads = K >> 2;
  const long long total = (long long)M * quads, plane = (long long)M * Kp;
  for (long long i = blockIdx.x * 256ll + threadIdx.x; i < total; i += gridDim.x * 256ll) {
    const int m = (int)(i / quads), k = (int)(i - (long long)m * quads) << 2;
    const float* src = x + (long long)m * ldx + k;
    float4 v;
    if (vec) v = *reinterpret_cast<const float4*>(src);
    else v = make_float4(src[0], src[1], src[2], src[3]);
    uint2 h, md, l;
    fs_cut(v.x, v.y, h.x, md.x, l.x);
    fs_cut(v.z, v.w, h.y, md.y, l.y);
    bf16* at = pieces + (long long)m * Kp + k;
    *reinterpret_cast<uint2*>(at) = h;
    *reinterpret_cast<uint2*>(at + plane) = md;
    *reinterpret_cast<uint2*>(at + 2 * plane) = l;
  }
}

// out = sum of the stretches' sums in order (+ bias).
template <int V>
__global__ void __launch_bounds__(256, 4) f32_fold_kernel(const SplitParams p, const float* partial) {
  KVB_KERNEL_PROLOGUE(KVB_TAG_GEMM_F32);
  const int pieces = p.N / V;
  const long long total = (long long)p.M * pieces, plane = (long long)p.M * p.N;
  const bool out16 = (p.ldo & 3) == 0 && aligned16(p.out);
  for (long long i = blockIdx.x * 256ll + threadIdx.x; i < total; i += gridDim.x * 256ll) {
    const int m = (int)(i / pieces), n = (int)(i - (long long)m * pieces) * V;
    const float* from = partial + (long long)m * p.N + n;
    float* const to = p.out + (long long)m * p.ldo + n;
    float sum[V];
#pragma unroll
    for (int c = 0; c < V; ++c) sum[c] = 0.0f;
#pragma unroll 4
    for (int s = 0; s < p.segments; ++s) {                 // 0 + the first sum is that sum (and a zero's sign is a plus)
      if constexpr (V == 4) {
        const float4 v = *reinterpret_cast<const float4*>(from + s * plane);
        sum[0] += v.x; sum[1] += v.y; sum[2] += v.z; sum[3] += v.w;
      } else {
        sum[0] += from[s * plane];
      }
    }
    bool finite = true;
#pragma unroll
    for (int c = 0; c < V; ++c) finite = finite && isfinite(sum[c]);
    if (!finite) {
      const float* rows[FS_AGAIN];
      float again[FS_AGAIN];
#pragma unroll
      for (int c = 0; c < FS_AGAIN; ++c) rows[c] = p.w + (long long)(n + (c < V ? c : 0)) * p.K;
      fs_by_fma(again, p.x + m * p.ldx, p.x16 != 0, rows, true, p.K);
#pragma unroll
      for (int c = 0; c < V; ++c)
        if (!isfinite(sum[c])) sum[c] = again[c];
    }
#pragma unroll
    for (int c = 0; c < V; ++c)
      if (p.bias != nullptr) sum[c] += p.bias[n + c];
    if (V == 4 && out16) {
      *reinterpret_cast<float4*>(to) = make_float4(sum[0], sum[1 % V], sum[2 % V], sum[3 % V]);
    } else {
#pragma unroll
      for (int c = 0; c < V; ++c) to[c] = sum[c];
    }
  }
}

template <int W>
__device__ __forceinline__ void fs_ld(unsigned taddr, float (&v)[W]) {      // W columns of this thread's lane
  unsigned* r = reinterpret_cast<unsigned*>(v);
  if constexpr (W == 8) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]) : "r"(taddr));
  } else if constexpr (W == 16) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                   "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]) : "r"(taddr));
  } else {
    kvb_tc5_ld32(taddr, v);
  }
}

template <int NT> struct SplitRing {
  // Warps that cut and warps that add.  Two groups of eight that cut in turn, with four that add, were slower for few rows as
  // well (56 us for 52 at one row, N 16384, K 3072): they leave a thread 88 registers.
  // The rows of a decode step cut in the block, by four more warps, instead of in a launch in front: 59 us for 52 at four rows,
  // N 16384, K 3072, 19.5 for 21.5 at N 3072, K 2048.
  static constexpr int CUT = 8, ADD = 8;
  static constexpr int THREADS = (CUT + ADD + 3) * 32;
  // stages of the two rings: what 227 KB hold
  static constexpr int X_BYTES = 3 * NT * FS_K * 2;
  static constexpr int WS = NT >= 128 ? 4 : NT >= 64 ? 5 : 6;
  static constexpr int BYTES = WS * FS_W_BYTES + 2 * X_BYTES + 512;
};

// NT rows of x a block (columns of the accumulators).
template <int NT>
__global__ void __launch_bounds__(SplitRing<NT>::THREADS, 1)
f32_split_kernel(const __grid_constant__ CUtensorMap w_map, const __grid_constant__ CUtensorMap x_map, const SplitParams p) {
  using Ring = SplitRing<NT>;
  constexpr int WS = Ring::WS, X_BYTES = Ring::X_BYTES, CUT = Ring::CUT, ADD = Ring::ADD;
  constexpr int CW = NT / (ADD / 4);                       // accumulator columns of a thread that adds
  extern __shared__ __align__(1024) unsigned char fs_dyn[];
  unsigned char* w_smem = fs_dyn;
  unsigned char* x_smem = w_smem + WS * FS_W_BYTES;        // two stages
  unsigned long long* w_full = reinterpret_cast<unsigned long long*>(x_smem + 2 * X_BYTES);   // [WS] weights landed
  unsigned long long* w_empty = w_full + WS;               // [WS] the warps that cut have read them
  // [2] a chunk may be multiplied: the weights' pieces lie in tensor memory (8 warps), the rows' have landed (their copy),
  // the accumulator has been read (ADD warps).  One barrier: every wait of the issuing warp is time the tensor pipe stands
  unsigned long long* ready = w_empty + WS;
  unsigned long long* done = ready + 2;                    // [2] a chunk's products are done: accumulator full, pieces read
  unsigned* tmem_slot = reinterpret_cast<unsigned*>(done + 2);
  int* abort_flag = reinterpret_cast<int*>(tmem_slot + 1);

  KvbTrace trace(KVB_TAG_GEMM_F32);
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  if (kvb_smem(fs_dyn) & 1023u) {                          // cannot happen with the alignment asked for; never run misaligned
    if (threadIdx.x == 0) atomicOr(p.status, KVB_STATUS_WAIT_TIMEOUT);
    return;
  }
  // row tiles fastest: the blocks that read the same weights run beside one another
  const int m0 = (int)(blockIdx.x % p.tiles_m) * NT;
  const int n0 = (int)(blockIdx.x / p.tiles_m % p.tiles_n) * FS_COLS;
  const int seg = (int)(blockIdx.x / p.tiles_m / p.tiles_n);
  const int chunk0 = seg * p.seg_chunks, count = min(p.seg_chunks, p.chunks - chunk0);   // at least one
  if (threadIdx.x == 0) {
    for (int s = 0; s < WS; ++s) { kvb_mbar_init(&w_full[s], 1); kvb_mbar_init(&w_empty[s], 8); }
    for (int s = 0; s < 2; ++s) { kvb_mbar_init(&ready[s], CUT + ADD + 1); kvb_mbar_init(&done[s], 1); }
    *abort_flag = 0;
    kvb_mbar_init_fence();
  }
  if (warp == CUT + ADD + 1) kvb_tc5_alloc(tmem_slot, 512u);
  kvb_tc5_fence_before();
  __syncthreads();
  kvb_tc5_fence_after();
  const unsigned tmem = __shfl_sync(0xffffffffu, *tmem_slot, 0);
  kvb_grid_launch_dependents();

  auto gave_up = [&] {
    atomicOr(p.status, KVB_STATUS_WAIT_TIMEOUT);
    atomicExch(abort_flag, 1);
  };
  auto aborted = [&] { return *reinterpret_cast<volatile int*>(abort_flag) != 0; };
  auto is_done = [&](int c) { return kvb_mbar_wait<FS_SPIN_LIMIT, 4096>(&done[c & 1], (c >> 1) & 1); };
  if (warp == CUT + ADD) {
    // ================= weights, as they are =================
    if (lane == 0) {
      int issued = 0;
      for (int c = 0; c < count; ++c) {
        const int s = c % WS;
        if (c >= WS && !kvb_mbar_wait<FS_SPIN_LIMIT, 4096>(&w_empty[s], ((c / WS) - 1) & 1)) { gave_up(); break; }
        if (aborted()) break;
        kvb_mbar_expect_tx(&w_full[s], FS_W_BYTES);
        kvb_tma_2d(w_smem + s * FS_W_BYTES, &w_map, (chunk0 + c) * FS_K, n0, &w_full[s]);
        kvb_tma_2d(w_smem + s * FS_W_BYTES + FS_W_BYTES / 2, &w_map, (chunk0 + c) * FS_K + FS_K / 2, n0, &w_full[s]);
        issued = c + 1;
      }
      if (aborted())                                       // let the copies in flight land before the block may exit
        for (int c = max(0, issued - WS); c < issued; ++c) kvb_mbar_wait<FS_SPIN_LIMIT, 4096>(&w_full[c % WS], (c / WS) & 1);
    }
  } else if (warp == CUT + ADD + 2) {
    // ================= the rows' pieces =================
    if (lane == 0) {
      kvb_grid_wait();                                     // the kernel in front wrote them
      int issued = 0;
      for (int c = 0; c < count; ++c) {
        if (c >= 2 && !is_done(c - 2)) { gave_up(); break; }
        if (aborted()) break;
        kvb_mbar_expect_tx(&ready[c & 1], X_BYTES);
        kvb_tma_3d(x_smem + (c & 1) * X_BYTES, &x_map, (chunk0 + c) * FS_K, m0, 0, &ready[c & 1]);
        issued = c + 1;
      }
      // given up: the barrier of the last copies may never complete (others count on it too), so they get the time that a
      // full wait takes instead
      if (aborted())
        for (int c = max(0, issued - 2); c < issued; ++c) kvb_mbar_wait<1u << 14, 0>(&ready[c & 1], (c >> 1) & 1);
    }
  } else if (warp == CUT + ADD + 1) {
    // ================= products: the whole warp, one lane issues =================
    const unsigned idesc = kvb_tc5_idesc(FS_COLS, NT, false), leader = kvb_elect();
    const unsigned long long x_desc = kvb_tc5_desc(kvb_smem(x_smem), 16, 1024);
    bool ok = true;
    int issued = 0;
    for (int c = 0; c < count; ++c) {
      const unsigned b = c & 1;
      ok = __all_sync(0xffffffffu, kvb_mbar_wait<FS_SPIN_LIMIT, 4096>(&ready[b], (c >> 1) & 1));
      if (!ok) break;
      kvb_tc5_fence_after();
      const unsigned acc = tmem + b * 128, a = tmem + FS_TMEM_W + b * 96;
      const unsigned long long x0 = x_desc + b * (X_BYTES / 16);
      constexpr int PIECE = NT * FS_K * 2 / 16;            // a piece of the rows, in the descriptor's units of 16 bytes
      // Pieces (weight, row), 0 the largest: small products first.  What the pieces' factors of 2^8 and 2^16 made of them is taken
      // back from sum to sum: the three smallest stand 2^16 too high, the next two 2^8.
      kvb_tc5_mma4_ts<8, 2>(acc, a + 64, x0, idesc, 0u, leader);
      kvb_tc5_mma4_ts<8, 2>(acc, a, x0 + 2 * PIECE, idesc, 1u, leader);
      kvb_tc5_mma4_ts<8, 2>(acc, a + 32, x0 + PIECE, idesc, 1u, leader);
      kvb_tc5_mma4_ts<8, 2, 8>(acc, a + 32, x0, idesc, 1u, leader);
      kvb_tc5_mma4_ts<8, 2>(acc, a, x0 + PIECE, idesc, 1u, leader);
      kvb_tc5_mma4_ts<8, 2, 8>(acc, a, x0, idesc, 1u, leader);
      kvb_tc5_commit_by(&done[b], leader);
      issued = c + 1;
    }
    if (!ok) {
      if (lane == 0) gave_up();                            // tensor memory is given back below: products in flight first
      if (issued > 0) is_done(issued - 1);
    }
    __syncwarp();
  } else if (warp < CUT) {
    // ================= cutting the weights =================
    const int half = warp >> 2, row = threadIdx.x & 127;   // half of the chunk's k
    const unsigned at0 = tmem + ((unsigned)((warp & 3) * 32) << 16) + FS_TMEM_W + half * 16;
    const unsigned char* const src0 = w_smem + half * (FS_W_BYTES / 2) + row * 128;
    float4 q[8];
    auto fetch = [&](int c) {
      const int s = c % WS;
      if (!__all_sync(0xffffffffu, kvb_mbar_wait<FS_SPIN_LIMIT, 4096>(&w_full[s], (c / WS) & 1))) return false;
#pragma unroll
      for (int i = 0; i < 8; ++i) q[i] = *reinterpret_cast<const float4*>(src0 + s * FS_W_BYTES + ((i ^ (row & 7)) << 4));
      return true;
    };
    bool ok = fetch(0);
    for (int c = 0; c < count && ok; ++c) {
      float piece[3][16];
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        unsigned h0, m0_, l0, h1, m1, l1;
        fs_cut(q[i].x, q[i].y, h0, m0_, l0);
        fs_cut(q[i].z, q[i].w, h1, m1, l1);
        piece[0][2 * i] = __uint_as_float(h0); piece[0][2 * i + 1] = __uint_as_float(h1);
        piece[1][2 * i] = __uint_as_float(m0_); piece[1][2 * i + 1] = __uint_as_float(m1);
        piece[2][2 * i] = __uint_as_float(l0); piece[2][2 * i + 1] = __uint_as_float(l1);
      }
      __syncwarp();
      if (lane == 0) kvb_mbar_arrive(&w_empty[c % WS]);
      if (c + 1 < count) ok = fetch(c + 1);                // on their way while the pieces are stored
      if (c >= 2 && ok) ok = __all_sync(0xffffffffu, is_done(c - 2));     // its products have read this stage
      if (!ok) break;
      kvb_tc5_fence_after();
      const unsigned at = at0 + (c & 1) * 96;
#pragma unroll
      for (int i = 0; i < 3; ++i) kvb_tc5_st16(at + i * 32, piece[i]);
      kvb_tc5_wait_st();
      kvb_tc5_fence_before();
      __syncwarp();
      if (lane == 0) kvb_mbar_arrive(&ready[c & 1]);
    }
    if (!ok && lane == 0) gave_up();
  } else {
    // ================= the sums =================
    const int half = (warp - CUT) >> 2, row = threadIdx.x & 127;       // of the accumulator's columns
    const unsigned from = tmem + ((unsigned)((warp & 3) * 32) << 16) + half * CW;
    if (lane == 0) {
      kvb_mbar_arrive(&ready[0]);                          // both accumulators are free
      if (count > 1) kvb_mbar_arrive(&ready[1]);
    }
    float sum[CW];
#pragma unroll
    for (int j = 0; j < CW; ++j) sum[j] = 0.0f;
    bool ok = true;
    for (int c = 0; c < count; ++c) {
      ok = __all_sync(0xffffffffu, is_done(c));
      if (!ok) break;
      kvb_tc5_fence_after();
      constexpr int W = CW < 16 ? CW : 16;
#pragma unroll
      for (int j = 0; j < CW; j += W) {
        float v[W];
        fs_ld<W>(from + (c & 1) * 128 + j, v);
        kvb_tc5_wait_ld();
#pragma unroll
        for (int i = 0; i < W; ++i) sum[j + i] += v[i];
      }
      kvb_tc5_fence_before();
      __syncwarp();
      if (lane == 0 && c + 2 < count) kvb_mbar_arrive(&ready[c & 1]);
    }
    if (ok) {
      const int n = n0 + row;
      kvb_grid_wait();                                     // `out` may be what the kernel in front still reads
      if (n < p.N) {
        float* const to = p.out + (p.segments > 1 ? (long long)seg * p.M * p.N : 0ll) + n;
        const float bias = p.bias != nullptr && p.segments == 1 ? p.bias[n] : 0.0f;
        unsigned long long again = 0;                      // outputs that are not finite
#pragma unroll
        for (int j = 0; j < CW; ++j) {
          const int m = m0 + half * CW + j;
          if (m < p.M) {
            if (!isfinite(sum[j])) again |= 1ull << j;
            to[(long long)m * p.ldo] = sum[j] + bias;
          }
        }
        if (p.segments > 1) again = 0;                     // the kernel that adds the stretches looks after these
        while (again) {
          int m[FS_AGAIN];
          const float* rows[FS_AGAIN];
          float value[FS_AGAIN];
#pragma unroll
          for (int r = 0; r < FS_AGAIN; ++r) {             // the last of them again where there are fewer
            m[r] = again ? m0 + half * CW + __ffsll((long long)again) - 1 : m[r > 0 ? r - 1 : 0];
            again &= again - 1;
            rows[r] = p.x + m[r] * p.ldx;
          }
          fs_by_fma(value, p.w + (long long)n * p.K, true, rows, p.x16 != 0, p.K);
#pragma unroll
          for (int r = 0; r < FS_AGAIN; ++r) to[(long long)m[r] * p.ldo] = value[r] + bias;
        }
      }
    } else if (lane == 0) {
      gave_up();
    }
  }
  kvb_tc5_fence_before();
  __syncthreads();
  if (warp == CUT + ADD + 1) {
    kvb_tc5_fence_after();
    kvb_tc5_dealloc(tmem, 512u);
  }
}

// ---- host side ------------------------------------------------------------------------------------------------------------
#define FS_MIN_K 2048
#define FS_MIN_N 128

// Stretches of K: the number whose blocks take the SMs least time, in chunks (a block costs about four beside its own), for
// one row tile and for two together.  A function of N and K alone, so that the order of the sums is.
static void split_segments(int N, int K, int* segments, int* seg_chunks) {
  const long long sms = kvb_sm_count() > 0 ? kvb_sm_count() : 148;
  const long long tiles = (N + FS_COLS - 1) / FS_COLS, chunks = (K + FS_K - 1) / FS_K;
  long long best = 0;
  for (long long s = 1; s <= 16 && s * 4 <= chunks; ++s) {
    const long long length = (chunks + s - 1) / s, count = (chunks + length - 1) / length;
    const long long cost = ((tiles * count + sms - 1) / sms + (2 * tiles * count + sms - 1) / sms) * (length + 4);
    if (best == 0 || cost < best) {
      best = cost;
      *segments = (int)count;
      *seg_chunks = (int)length;
    }
  }
}
// Whether w [N, K] takes this kernel, whatever the rows: the order of the sums may not depend on them.  Microseconds, this one and
// gemm_f32.cu, in a captured run of calls on different weights.  One row: K 2048: N 128 8.4 and 15.3, N 1024 9.6 and 15.4, N 2048
// 12.5 and 15.6, N 3072 14.9 and 16.1, N 5120 16.0 and 18.4, N 16384 31.4 and 36.9; K 3072: N 128 9.0 and 22.4, N 3072 15.2 and
// 23.6, N 16384 42.2 and 53.7; below K 2048 with launches of their own: N 2048: K 512 15 and 10, K 1024 15.4 and 14.4, K 1280 15.4
// and 16.4; N 4096, K 1280 19.5 and 16.4.  A single row loses where the other kernel's blocks of 16 columns just fill a round
// of the GPU (9,472 columns, four blocks an SM): K 2048: N 6400 19.5 and 18.5, N 8192 20.3 and 19.1, N 9472 22.5 and 19.2; K 2560: N
// 6912 26.1 and 22.7; K 3072: N 6912 29.2 and 27.2; K 2048, N 26624 55.8 and 53.9.  With more rows it does not: N 8192, K 2048: 2
// rows 20.4 and 21.1, 8 rows 21.6 and 38, 64 rows 25 and 102, 256 rows 54 and 242; N 6912, K 2560: 8 rows 27 and 44.
static bool split_takes(const void* w, int N, int K) {
  return K % 4 == 0 && aligned16(w) && K >= FS_MIN_K && N >= FS_MIN_N;
}
extern "C" int kvb_gemm_f32_split_min_k() { return FS_MIN_K; }
static int split_lot(int M, int N, int segments) {          // rows whose sums of stretches fit the scratch's bound
  if (segments == 1) return M;
  const long long rows = FS_MAX_PARTIAL_FLOATS / ((long long)segments * N) / 128 * 128;
  return (int)(rows < 128 ? (M < 128 ? M : 128) : rows < M ? rows : M);
}

// Bytes of scratch that kvb_gemm_f32_split needs for this product (16-byte aligned); 0: the product takes kvb_gemm_f32.
extern "C" long long kvb_gemm_f32_split_scratch(const void* w, int M, int N, int K) {
  if (M <= 0 || N <= 0 || K <= 0 || !split_takes(w, N, K)) return 0;
  int segments, seg_chunks;
  split_segments(N, K, &segments, &seg_chunks);
  const long long lot = split_lot(M, N, segments), Kp = (K + 7) / 8 * 8;
  return (3 * lot * Kp * 2 + 15) / 16 * 16 + (segments > 1 ? segments * lot * N * 4 : 0);
}

// Kernels that kvb_gemm_f32_split launches for a product that takes it.
extern "C" int kvb_gemm_f32_split_launches(int M, int N, int K) {
  int segments, seg_chunks;
  split_segments(N, K, &segments, &seg_chunks);
  const int lot = split_lot(M, N, segments);
  int launches = 0;
  for (int first = 0; first < M; first += lot) launches += segments > 1 ? 3 : 2;   // cutting, products, adding
  return launches;
}

template <int NT>
static int launch_split(const CUtensorMap& w_map, const CUtensorMap& x_map, const SplitParams& p, cudaStream_t stream) {
  KVB_CHECK_CUDA(cudaFuncSetAttribute(f32_split_kernel<NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, SplitRing<NT>::BYTES));
  const long long blocks = (long long)p.tiles_m * p.tiles_n * p.segments;
  KVB_REQUIRE(blocks <= 0x7fffffffll, "gemm_f32: too many tiles for one launch");
  KVB_CHECK_CUDA(kvb_launch((f32_split_kernel<NT>), dim3((unsigned)blocks), dim3(SplitRing<NT>::THREADS), SplitRing<NT>::BYTES, stream, true,
                            w_map, x_map, p));
  return 0;
}

extern "C" int kvb_gemm_f32_split(float* out, const float* x, const float* w, const float* bias, int M, int N, int K,
                                  long long ldx, long long ldo, void* scratch, cudaStream_t stream) {
  if (M == 0 || N == 0) return 0;
  KVB_REQUIRE(K > 0 && split_takes(w, N, K) && scratch != nullptr && aligned16(scratch), "gemm_f32: the product does not take pieces");
  KvbEncodeTiledFn encode = kvb_encode_tiled_fn();
  KVB_REQUIRE(encode != nullptr, "gemm_f32: the driver does not export cuTensorMapEncodeTiled");
  SplitParams p = {};
  p.status = kvb_status_word();
  KVB_REQUIRE(p.status != nullptr, "gemm_f32: no status word");
  split_segments(N, K, &p.segments, &p.seg_chunks);
  p.chunks = (K + FS_K - 1) / FS_K;
  p.tiles_n = (N + FS_COLS - 1) / FS_COLS;
  p.N = N; p.K = K; p.w = w; p.ldx = ldx;
  p.bias = p.segments == 1 ? bias : nullptr;
  const cuuint32_t elem[3] = {1, 1, 1};
  alignas(64) CUtensorMap w_map, x_map;
  {
    const cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)N};
    const cuuint64_t strides[1] = {(cuuint64_t)K * 4};
    const cuuint32_t box[2] = {FS_K / 2, FS_COLS};
    KVB_REQUIRE(encode(&w_map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float*>(w), dims, strides, box, elem,
                       CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                       CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS,
                "gemm_f32: cuTensorMapEncodeTiled failed for the weights");
  }
  const int lot = split_lot(M, N, p.segments), Kp = (K + 7) / 8 * 8;
  bf16* pieces = (bf16*)scratch;
  float* partial = (float*)((char*)scratch + (3ll * lot * Kp * 2 + 15) / 16 * 16);
  const long long fill = 8ll * (kvb_sm_count() > 0 ? kvb_sm_count() : 148);
  for (int first = 0; first < M; first += lot) {
    const int rows = M - first < lot ? M - first : lot;
    p.M = rows;
    p.x = x + (long long)first * ldx;
    p.out = p.segments > 1 ? partial : out + (long long)first * ldo;
    p.ldo = p.segments > 1 ? N : ldo;
    p.x16 = ldx % 4 == 0 && aligned16(p.x) ? 1 : 0;
    const long long cut = ((long long)rows * (K / 4) + 255) / 256;
    KVB_CHECK_CUDA(kvb_launch(f32_pieces_kernel, dim3((unsigned)(cut < fill ? cut : fill)), dim3(256), 0, stream, true, pieces, p.x, rows, K,
                              Kp, ldx, p.x16));
    // tiles of 64 rows where 128 would hold many rows that are not there (a chunk of 64 rows costs half)
    const int nt = rows <= 16 ? 16 : rows <= 32 ? 32 : (rows + 63) / 64 * 64 < (rows + 127) / 128 * 128 ? 64 : 128;
    p.tiles_m = (rows + nt - 1) / nt;
    const cuuint64_t dims[3] = {(cuuint64_t)K, (cuuint64_t)rows, 3};
    const cuuint64_t strides[2] = {(cuuint64_t)Kp * 2, (cuuint64_t)rows * Kp * 2};
    const cuuint32_t box[3] = {FS_K, (cuuint32_t)nt, 3};
    KVB_REQUIRE(encode(&x_map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, pieces, dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
                       CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS,
                "gemm_f32: cuTensorMapEncodeTiled failed for the rows");
    const int rc = nt == 16 ? launch_split<16>(w_map, x_map, p, stream) : nt == 32 ? launch_split<32>(w_map, x_map, p, stream)
                 : nt == 64 ? launch_split<64>(w_map, x_map, p, stream) : launch_split<128>(w_map, x_map, p, stream);
    if (rc != 0) return rc;
    if (p.segments > 1) {
      const bool four = N % 4 == 0;
      const long long folds = ((long long)rows * (four ? N / 4 : N) + 255) / 256;
      const dim3 grid((unsigned)(folds < fill ? folds : fill));
      SplitParams f = p;
      f.out = out + (long long)first * ldo;
      f.ldo = ldo;
      f.bias = bias;
      KVB_CHECK_CUDA(four ? kvb_launch((f32_fold_kernel<4>), grid, dim3(256), 0, stream, true, f, (const float*)partial)
                          : kvb_launch((f32_fold_kernel<1>), grid, dim3(256), 0, stream, true, f, (const float*)partial));
    }
  }
  KVB_CHECK_LAUNCH();
  return 0;
}

KVB_TRACE_TU(gemm_f32_tc5)
