// True 32-bit linear layer: out[m, n] = sum_k x[m, k] * w[n, k] (+ bias[n]), FMA on the CUDA
// cores only, no tensor cores and no reduced-precision mode.  Matrices with K from 2,048 on take gemm_f32_tc5.cu, whatever
// the rows.
//
// Every output element is one accumulator that takes its products in ascending k, so its value
// does not depend on M, on the kernel or the tile it falls in, or on the rest of the batch: the
// 32-bit path is bit-identical under any cutting of the work.  Every M, N, K is accepted (edges
// are zero-filled in shared memory, adding exact zeros).
//
// Two kernels:
//   gemm_f32_tile: a TM x TN tile a block, RM x RN outputs a thread, K in slabs of 16 through two
//     stages of shared memory, the next slab on its way from memory into registers meanwhile.
//     What bounds it is the rate of the FMA units and of the shared-memory reads that feed them:
//     8 x 8 outputs a thread take 4 reads for 64 FMA, smaller patches more, but smaller tiles leave
//     fewer SMs idle in the last round.  256 rows on B200: N 16384, K 3072 at 41.8 TFLOP/s (one tile
//     of 64 x 64 with single-buffered slabs, which this took the place of: 20.4); N 3072, K 3072 at
//     29.9 (14.4); N 3072, K 8192 at 30.6 (14.6).
//   gemm_f32_rows: up to 16 rows (a decode step).  A block owns 16 columns, a thread one output;
//     the weights stream through four stages of asynchronous copies.  What bounds it is the pass
//     over the weights, or, for few columns, the chain of K dependent FMA of an output.  8 rows, N 5120,
//     K 3072: 50 us against 173 for the smallest tile; one row, N 16384, K 2048: 42 us against 119.
#include "common.cuh"

#define GK 16                 // k of a slab (tile kernel)
#define GR_COLS 16            // columns of a block (rows kernel)
#define GR_MAX_ROWS 16
#define GR_K 128              // k of a stage (rows kernel)
#define GR_STAGES 4
#define GR_LD (GR_K + 4)      // rows of a stage start 4 banks apart: eight lanes' 16-byte reads cover all banks

struct GemmF32Params {
  float* out; const float* x; const float* w; const float* bias;
  int M, N, K;
  long long ldx, ldo;
};

// Two products and sums in one instruction, each rounded as fmaf rounds them: the FMA units' rate is the same, the
// instruction slots that are left over go to the shared-memory reads (41.8 against 38.2 TFLOP/s with fmaf).
__device__ __forceinline__ unsigned long long fma_pair(unsigned long long a, unsigned long long b, unsigned long long c) {
  unsigned long long d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ unsigned long long twice(float a) {
  unsigned long long d;
  asm("mov.b64 %0, {%1, %1};" : "=l"(d) : "r"(__float_as_uint(a)));
  return d;
}

// VEC: K and ldx multiples of four, x and w on 16-byte boundaries.
template <int TM, int TN, int RM, int RN, bool VEC>
__global__ void __launch_bounds__(TM / RM * (TN / RN), TM * TN >= 128 * 128 ? 2 : 1)
gemm_f32_tile_kernel(GemmF32Params p) {
  KVB_KERNEL_PROLOGUE(KVB_TAG_GEMM_F32);
  constexpr int THREADS = TM / RM * (TN / RN), TX = TN / RN;
  constexpr int LM = TM + 4, LN = TN + 4;
  constexpr int XPT = TM * GK / 4 / THREADS, WPT = TN * GK / 4 / THREADS;      // four neighbouring k a piece
  static_assert(XPT * THREADS * 4 == TM * GK && WPT * THREADS * 4 == TN * GK, "a slab is whole pieces a thread");
  static_assert(RM % 4 == 0 && RN % 4 == 0 && TX % 8 == 0 && TM / RM % 4 == 0, "patches are quads, warps 4 x 8 threads");
  __shared__ __align__(16) float xs[2][GK][LM];
  __shared__ __align__(16) float ws[2][GK][LN];
  const int m0 = blockIdx.y * TM, n0 = blockIdx.x * TN;
  // a warp is 4 x 8 threads, and neighbouring lanes share a row: the 16-byte reads of a warp then touch few distinct
  // lines next to one another, which the shared memory serves in fewer turns
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int tx = warp % (TX / 8) * 8 + ((lane >> 1) & 7), ty = warp / (TX / 8) * 4 + (lane & 1) + 2 * (lane >> 4);
  unsigned long long acc[RM][RN / 2];                   // pairs of neighbouring columns
#pragma unroll
  for (int i = 0; i < RM; ++i)
#pragma unroll
    for (int j = 0; j < RN / 2; ++j) acc[i][j] = 0;

  float4 xr[XPT], wr[WPT];
  auto piece = [&](const float* row, bool inside, int k) {
    float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (!inside || k >= p.K) return v;
    if (VEC) return *reinterpret_cast<const float4*>(row + k);       // K is a multiple of four
    v.x = row[k];
    if (k + 1 < p.K) v.y = row[k + 1];
    if (k + 2 < p.K) v.z = row[k + 2];
    if (k + 3 < p.K) v.w = row[k + 3];
    return v;
  };
  auto load = [&](int k0) {
#pragma unroll
    for (int r = 0; r < XPT; ++r) {
      const int idx = threadIdx.x + r * THREADS, m = m0 + idx / (GK / 4), k = k0 + idx % (GK / 4) * 4;
      xr[r] = piece(p.x + (size_t)(m < p.M ? m : 0) * p.ldx, m < p.M, k);
    }
#pragma unroll
    for (int r = 0; r < WPT; ++r) {
      const int idx = threadIdx.x + r * THREADS, n = n0 + idx / (GK / 4), k = k0 + idx % (GK / 4) * 4;
      wr[r] = piece(p.w + (size_t)(n < p.N ? n : 0) * p.K, n < p.N, k);
    }
  };
  auto store = [&](int stage) {
#pragma unroll
    for (int r = 0; r < XPT; ++r) {
      const int idx = threadIdx.x + r * THREADS, row = idx / (GK / 4), k = idx % (GK / 4) * 4;
      xs[stage][k][row] = xr[r].x; xs[stage][k + 1][row] = xr[r].y; xs[stage][k + 2][row] = xr[r].z; xs[stage][k + 3][row] = xr[r].w;
    }
#pragma unroll
    for (int r = 0; r < WPT; ++r) {
      const int idx = threadIdx.x + r * THREADS, row = idx / (GK / 4), k = idx % (GK / 4) * 4;
      ws[stage][k][row] = wr[r].x; ws[stage][k + 1][row] = wr[r].y; ws[stage][k + 2][row] = wr[r].z; ws[stage][k + 3][row] = wr[r].w;
    }
  };
  // a thread's rows are quads TM / (RM / 4) apart and its columns quads TN / (RN / 4) apart: the lanes of a warp
  // read neighbouring quads
  constexpr int MS = TM / (RM / 4), NS = TN / (RN / 4);
  load(0);
  store(0);
  __syncthreads();
  int stage = 0;
  for (int k0 = 0; k0 < p.K; k0 += GK, stage ^= 1) {
    const bool more = k0 + GK < p.K;
    if (more) load(k0 + GK);
#pragma unroll
    for (int kk = 0; kk < GK; ++kk) {
      unsigned long long a[RM], b[RN / 2];
#pragma unroll
      for (int i = 0; i < RM / 4; ++i) {
        const float4 v = *reinterpret_cast<const float4*>(&xs[stage][kk][i * MS + ty * 4]);
        a[4 * i] = twice(v.x); a[4 * i + 1] = twice(v.y); a[4 * i + 2] = twice(v.z); a[4 * i + 3] = twice(v.w);
      }
#pragma unroll
      for (int j = 0; j < RN / 4; ++j) {
        const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(&ws[stage][kk][j * NS + tx * 4]);
        b[2 * j] = v.x; b[2 * j + 1] = v.y;
      }
#pragma unroll
      for (int i = 0; i < RM; ++i)
#pragma unroll
        for (int j = 0; j < RN / 2; ++j) acc[i][j] = fma_pair(a[i], b[j], acc[i][j]);
    }
    if (more) store(stage ^ 1);           // the last readers of that stage passed the barrier below one slab ago
    __syncthreads();
  }
  const bool out16 = (p.ldo & 3) == 0 && (p.N & 3) == 0 && ((uintptr_t)p.out & 15) == 0;
#pragma unroll
  for (int i = 0; i < RM; ++i) {
    const int m = m0 + i / 4 * MS + ty * 4 + i % 4;
    if (m >= p.M) continue;
#pragma unroll
    for (int j = 0; j < RN; j += 4) {
      const int n = n0 + j / 4 * NS + tx * 4;
      float* at = p.out + (size_t)m * p.ldo + n;
      float v[4];
#pragma unroll
      for (int c = 0; c < 4; ++c)
        v[c] = __uint_as_float((unsigned)(acc[i][(j + c) / 2] >> (c % 2 * 32))) + (p.bias && n + c < p.N ? p.bias[n + c] : 0.0f);
      if (out16 && n < p.N) {
        *reinterpret_cast<float4*>(at) = make_float4(v[0], v[1], v[2], v[3]);
      } else {
#pragma unroll
        for (int c = 0; c < 4; ++c)
          if (n + c < p.N) at[c] = v[c];
      }
    }
  }
}

template <bool VEC>
__device__ __forceinline__ void gemm_rows_copy(float* dst, const float* src, int valid) {   // `valid` floats, else zeros
  const unsigned to = (unsigned)__cvta_generic_to_shared(dst);
  if (VEC) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(to), "l"(src), "r"(valid > 0 ? 16 : 0));
  } else {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(to), "l"(src), "r"(valid > 0 ? 4 : 0));
  }
}

// ROWS: 8 or 16 rows of x a block holds (M of them real).
template <int ROWS, bool VEC>
__global__ void __launch_bounds__(ROWS * GR_COLS)
gemm_f32_rows_kernel(GemmF32Params p) {
  KVB_KERNEL_PROLOGUE(KVB_TAG_GEMM_F32);
  extern __shared__ __align__(16) float stages[];               // [GR_STAGES][GR_COLS + ROWS][GR_LD]
  constexpr int THREADS = ROWS * GR_COLS, STAGE = (GR_COLS + ROWS) * GR_LD, N = VEC ? 4 : 1;
  const int n0 = blockIdx.x * GR_COLS, col = threadIdx.x % GR_COLS, row = threadIdx.x / GR_COLS;
  const int live = GR_COLS + p.M;                               // rows of a stage that hold anything
  auto fetch = [&](int stage, int k0) {
    for (int e = threadIdx.x; e < live * (GR_K / N); e += THREADS) {
      const int r = e / (GR_K / N), k = k0 + e % (GR_K / N) * N;
      const bool weight = r < GR_COLS;
      const int valid = k < p.K && (!weight || n0 + r < p.N) ? N : 0;
      const float* base = weight ? p.w + (size_t)(n0 + r) * p.K : p.x + (size_t)(r - GR_COLS) * p.ldx;
      gemm_rows_copy<VEC>(stages + stage * STAGE + r * GR_LD + (k - k0), valid ? base + k : p.w, valid);
    }
  };
#pragma unroll
  for (int s = 0; s < GR_STAGES - 1; ++s) {
    if (s * GR_K < p.K) fetch(s, s * GR_K);
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  }
  float acc = 0.0f;
  int stage = 0;
  for (int k0 = 0; k0 < p.K; k0 += GR_K) {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(GR_STAGES - 2) : "memory");
    __syncthreads();                                            // this stage is there; the one behind it is read out
    const int ahead = k0 + (GR_STAGES - 1) * GR_K;
    if (ahead < p.K) fetch((stage + GR_STAGES - 1) % GR_STAGES, ahead);
    asm volatile("cp.async.commit_group;\n" ::: "memory");
    if (row < p.M) {
      const float* w = stages + stage * STAGE + col * GR_LD;
      const float* x = stages + stage * STAGE + (GR_COLS + row) * GR_LD;
      const int pieces = min(GR_K, p.K - k0 + 3) >> 2;          // a last piece's missing entries are zeros
#pragma unroll 8
      for (int i = 0; i < pieces; ++i) {
        const float4 a = *reinterpret_cast<const float4*>(x + 4 * i), b = *reinterpret_cast<const float4*>(w + 4 * i);
        acc = fmaf(a.x, b.x, acc);
        acc = fmaf(a.y, b.y, acc);
        acc = fmaf(a.z, b.z, acc);
        acc = fmaf(a.w, b.w, acc);
      }
    }
    stage = (stage + 1) % GR_STAGES;
  }
  asm volatile("cp.async.wait_group 0;\n" ::: "memory");
  const int n = n0 + col;
  if (row < p.M && n < p.N) p.out[(size_t)row * p.ldo + n] = acc + (p.bias ? p.bias[n] : 0.0f);
}

template <int ROWS, bool VEC>
static cudaError_t launch_gemm_rows(const GemmF32Params& p, cudaStream_t stream) {
  constexpr int smem = GR_STAGES * (GR_COLS + ROWS) * GR_LD * (int)sizeof(float);
  const cudaError_t err = cudaFuncSetAttribute(gemm_f32_rows_kernel<ROWS, VEC>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (err != cudaSuccess) return err;
  return kvb_launch((gemm_f32_rows_kernel<ROWS, VEC>), dim3((p.N + GR_COLS - 1) / GR_COLS), dim3(ROWS * GR_COLS), smem, stream,
                    true, p);
}

template <int TM, int TN, int RM, int RN>
static cudaError_t launch_gemm_tile(const GemmF32Params& p, bool vec, cudaStream_t stream) {
  const dim3 grid((p.N + TN - 1) / TN, (p.M + TM - 1) / TM), block(TM / RM * (TN / RN));
  return vec ? kvb_launch((gemm_f32_tile_kernel<TM, TN, RM, RN, true>), grid, block, 0, stream, true, p)
             : kvb_launch((gemm_f32_tile_kernel<TM, TN, RM, RN, false>), grid, block, 0, stream, true, p);
}

extern "C" int kvb_gemm_f32(float* out, const float* x, const float* w, const float* bias, int M,
                            int N, int K, long long ldx, long long ldo, cudaStream_t stream) {
  if (M == 0 || N == 0) return 0;
  KVB_REQUIRE(K > 0, "gemm_f32: K must be positive");
  KVB_REQUIRE((M + 63) / 64 <= 65535, "gemm_f32: too many rows for one launch");
  const GemmF32Params p = {out, x, w, bias, M, N, K, ldx, ldo};
  const bool vec = K % 4 == 0 && ldx % 4 == 0 && aligned16(x) && aligned16(w);
  cudaError_t err;
  if (M <= GR_MAX_ROWS) {
    // a tile of 32 rows would be half empty or more, and few tiles cover the columns: see the rates above
    if (M <= 8) err = vec ? launch_gemm_rows<8, true>(p, stream) : launch_gemm_rows<8, false>(p, stream);
    else err = vec ? launch_gemm_rows<16, true>(p, stream) : launch_gemm_rows<16, false>(p, stream);
  } else {
    // The SMs work through the tiles in rounds of one tile each, and one or two tiles at a time do not fill an SM's
    // FMA units.  Microseconds at K = 2048 as measured (other K in proportion): 128 x 128 tiles 266 for a lone round,
    // else 210 a round; 64 x 64 tiles 58 a round, no less than 2.2 rounds; 32 x 64 tiles 38, no less than 2.7.
    // 77 x 4096: 266, 134 and 102; 256 x 3072: 257, 129 and 108; 256 x 16384: 425, 412 and 517; 1000 x 4096: 419, 399
    // and 463.
    const long long sms = kvb_sm_count() > 0 ? kvb_sm_count() : 148;
    auto rounds = [&](int tm, int tn) {
      const long long blocks = (long long)((M + tm - 1) / tm) * ((N + tn - 1) / tn);
      return (double)((blocks + sms - 1) / sms);
    };
    const double large = rounds(128, 128) < 2 ? 266.0 : 210.0 * rounds(128, 128);
    const double middle = 58.0 * (rounds(64, 64) < 2.2 ? 2.2 : rounds(64, 64));
    const double small = 38.0 * (rounds(32, 64) < 2.7 ? 2.7 : rounds(32, 64));
    if (large <= middle && large <= small) err = launch_gemm_tile<128, 128, 8, 8>(p, vec, stream);
    else if (middle <= small || (M + 31) / 32 > 65535) err = launch_gemm_tile<64, 64, 8, 4>(p, vec, stream);
    else err = launch_gemm_tile<32, 64, 4, 4>(p, vec, stream);
  }
  KVB_CHECK_CUDA(err);
  KVB_CHECK_LAUNCH();
  return 0;
}

KVB_TRACE_TU(gemm_f32)
