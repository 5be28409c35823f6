// The scan over a request's tokens of mixers that carry a matrix-valued state per request and head, everything in
// 32-bit.  A template: each source file that launches a mode makes its own kernels of it.
//
//   state_scan: per (request, head) a state S [D, V] (32-bit, one row of `state` per state slot) runs
//   over the request's tokens of this step in order.
//     decay per key channel (gated linear attention):
//         S <- diag(a_t) S + k_t v_t^T,                 o_t = S^T q_t
//         with a_t = sigmoid(z_t)^(1/tau) and q_t scaled by `q_scale`, as `gla_prepare` left them (32-bit);
//     delta rule with one decay per head:
//         S <- g_t S;  u = beta_t (v_t - S^T k_t);  S <- S + k_t u^T;  o_t = S^T q_t
//         with q_t, k_t, v_t, beta_t, g_t as `conv_prepare` left them (32-bit).
//     one fixed decay a head (lightning attention):
//         S <- a_h S + k_t v_t^T,                       o_t = S^T q_t
//         with q_t = silu(.) * q_scale, k_t = silu(.) and v_t = silu(.) as `lightning_prepare` left them (32-bit),
//         a_h a constant of the model;
//     one decay and one step size a head and token (selective state space):
//         S <- g_t S + B_t (dt_t x_t)^T,                o_t = S^T C_t + D_h x_t
//         with B_t, C_t (one of each for a group of heads), x_t, dt_t, g_t as `ssm_prepare` (state_space.cu) left them;
//   S is kept column by column ([H, V, D] in the state row: a column's D rows lie together).  A column is shared
//   by RSPLIT lanes of a warp, 32 / RSPLIT apart (8 or 16 rows each, in registers, loaded and stored as 16-byte
//   pieces); a thread holds those rows of one to four neighbouring columns; a block owns 128 / RSPLIT (times these) columns of
//   one (request, head).  The launch picks the shape (see scan_shape).
//   Columns never exchange anything, and a sum over a column's rows is taken in one fixed order (scan_eight) whatever the
//   shape, so any cut of a request into steps and any batch it runs in give the same bits.  The tokens' vectors (32-bit: q, k,
//   and the decays or beta and gate) come through stages of shared memory, by TMA where a map describes them
//   (state_scan_tma), else by cp.async.  The read-outs' sums over a column's threads are taken for eight tokens at once, off
//   the chain that carries S from token to token.
#pragma once

#include <stdlib.h>

#include "common.cuh"
#include "sm100.cuh"

#define SCAN_THREADS 128
#define SCAN_SM_BYTES (228 * 1024)     // shared memory of an SM; a block's share comes with 1 KB on top

__device__ __forceinline__ void scan_copy16(float* dst, const float* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src));
}
__device__ __forceinline__ void scan_copy4(float* dst, const float* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src));
}
__device__ __forceinline__ void scan_copies_done() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

// Two neighbouring rows of a column (or the same number twice) in one register pair; an instruction rounds each half as
// the plain one does, so the state has the same bits, and takes one issue slot for both.
typedef unsigned long long ScanPair;
__device__ __forceinline__ ScanPair scan_pair(float lo, float hi) {
  ScanPair d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "r"(__float_as_uint(lo)), "r"(__float_as_uint(hi)));
  return d;
}
__device__ __forceinline__ float scan_lo(ScanPair a) { return __uint_as_float((unsigned)a); }
__device__ __forceinline__ float scan_hi(ScanPair a) { return __uint_as_float((unsigned)(a >> 32)); }
__device__ __forceinline__ ScanPair scan_mul(ScanPair a, ScanPair b) {
  ScanPair d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ ScanPair scan_fma(ScanPair a, ScanPair b, ScanPair c) {
  ScanPair d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}

// Two rows of a column an instruction, eight rows: even and odd ones in order, then both together.  A sum over a column's rows
// is taken of such eights, and these are added as a tree over their numbers (n with n ^ 1, then with n ^ 2, ...): inside a
// thread for those it holds, by shuffles between the threads of a column.  The result has the same bits for every DREG and
// CPT, so a launch may pick both by how many columns it has.
__device__ __forceinline__ float scan_eight(const ScanPair* s, const ulonglong2& w0, const ulonglong2& w1) {
  const ScanPair sum = scan_fma(s[3], w1.y, scan_fma(s[2], w1.x, scan_fma(s[1], w0.y, scan_mul(s[0], w0.x))));
  return scan_lo(sum) + scan_hi(sum);
}

// What a token brings a thread: its columns' values (twice), q, k, decays of its rows.
template <int MODE, int J, int CPT>
struct ScanVectors {
  ScanPair v[CPT];
  ulonglong2 k4[J], a4[J], q4[J];
  float first, second;                              // beta and g, or dt and g
};

// One token: the state's step and this thread's part of the read-out of each of its columns.
template <int MODE, int DREG, int RSPLIT, int CPT>
__device__ __forceinline__ void scan_token(ScanPair (&S)[CPT][DREG / 2], ScanVectors<MODE, DREG / 4, CPT>& n, ScanPair head_decay,
                                           float (&o_own)[CPT]) {
  constexpr int J = DREG / 4, BESIDE = 32 / RSPLIT;
  if (MODE != 1) {
    ScanPair decay = MODE == 2 ? head_decay : 0;
    if (MODE == 3) {
      const float dt = n.first, g = n.second;
      decay = scan_pair(g, g);
#pragma unroll
      for (int cc = 0; cc < CPT; ++cc) n.v[cc] = scan_mul(scan_pair(dt, dt), n.v[cc]);
    }
#pragma unroll
    for (int j = 0; j < J; ++j) {
      ulonglong2 a4 = make_ulonglong2(decay, decay);
      if (MODE == 0) a4 = n.a4[j];
#pragma unroll
      for (int cc = 0; cc < CPT; ++cc) {
        ScanPair* s = &S[cc][2 * j];
        s[0] = scan_fma(n.k4[j].x, n.v[cc], scan_mul(a4.x, s[0]));
        s[1] = scan_fma(n.k4[j].y, n.v[cc], scan_mul(a4.y, s[1]));
      }
    }
  } else {
    const float beta = n.first, g = n.second;
    const ScanPair decay = scan_pair(g, g);
    float dot[CPT];
#pragma unroll
    for (int cc = 0; cc < CPT; ++cc) {
#pragma unroll
      for (int i = 0; i < DREG / 2; ++i) S[cc][i] = scan_mul(decay, S[cc][i]);
      dot[cc] = scan_eight(&S[cc][0], n.k4[0], n.k4[1]);
      if constexpr (J == 4) dot[cc] += scan_eight(&S[cc][4], n.k4[2], n.k4[3]);
    }
#pragma unroll
    for (int m = 1; m < RSPLIT; m <<= 1)
#pragma unroll
      for (int cc = 0; cc < CPT; ++cc) dot[cc] += __shfl_xor_sync(0xffffffffu, dot[cc], m * BESIDE);
#pragma unroll
    for (int cc = 0; cc < CPT; ++cc) {
      const float u1 = beta * (scan_lo(n.v[cc]) - dot[cc]);
      const ScanPair u = scan_pair(u1, u1);
#pragma unroll
      for (int j = 0; j < J; ++j) {
        ScanPair* s = &S[cc][2 * j];
        s[0] = scan_fma(n.k4[j].x, u, s[0]);
        s[1] = scan_fma(n.k4[j].y, u, s[1]);
      }
    }
  }
#pragma unroll
  for (int cc = 0; cc < CPT; ++cc) {
    o_own[cc] = scan_eight(&S[cc][0], n.q4[0], n.q4[1]);
    if constexpr (J == 4) o_own[cc] += scan_eight(&S[cc][4], n.q4[2], n.q4[3]);
  }
}

// The tree over a column's threads for N sums at once: a pair of threads shares the work of a level, either keeps half of the
// entries, hands the other half over and adds what it is handed (31 exchanges for 32 entries of 32 threads, not 160).  At
// the end a thread holds N / RSPLIT entries (at least one) at the front of `sums`; returns the number of the first.
template <int RSPLIT, int N>
__device__ __forceinline__ int scan_exchange(float (&sums)[N], int part) {
  int entry = 0;
#pragma unroll
  for (int m = 1, half = N / 2; m < RSPLIT; m <<= 1, half >>= 1) {
    if (half > 0) {
      const bool upper = (part & m) != 0;
      if (upper) entry += half;
#pragma unroll
      for (int i = 0; i < half; ++i) {
        const float keep = upper ? sums[i + half] : sums[i], give = upper ? sums[i] : sums[i + half];
        sums[i] = keep + __shfl_xor_sync(0xffffffffu, give, m * (32 / RSPLIT));
      }
    } else {
      sums[0] += __shfl_xor_sync(0xffffffffu, sums[0], m * (32 / RSPLIT));
    }
  }
  return entry;
}

struct ScanParams {
  // 32-bit vectors per token: q and k [D] of head h / kv_share, and (decay per key channel) the decays a [D]
  // of head h, each at base + t * vec_token + head * D
  const float* q; const float* k; const float* a;
  long long vec_token;
  int vec16;                                // every vector starts on a 16-byte boundary and D is a multiple of 4
  int state16;                              // so does every column of S in the state rows
  const void* v; long long v_token;         // values [V] of head h at v + t * v_token + h * V (elements)
  const float* beta; const float* gate;     // [T, H] with row stride bg_stride (delta rule: beta, g; state space: dt, g)
  const float* skip;                        // [H]: D (state space)
  long long bg_stride;
  float* out;                               // [T, H, V]
  float* state;                             // [slots, state_stride]; this mixer's S at state_offset, [H, V, D]
  long long state_stride, state_offset;
  const int* query_start; const int* state_slots;
  int heads, kv_share, D, V;
  int* status;
};

// MODE 0: decay per key channel; MODE 1: delta rule; MODE 2: one fixed decay a head (p.a[h]); MODE 3: one decay and
// step size a head and token, D_h x_t added to the read-out.  RSPLIT threads a column of S, DREG rows each; a thread
// holds those rows of CPT neighbouring columns (one load of q, k and the decays then serves CPT columns, and the
// columns' chains of dependent instructions run interleaved); BATCH tokens a stage of shared memory.
template <typename TV, int MODE, int DREG, int RSPLIT, int CPT, int BATCH>
// (brief: every block's state in flight counts; keys of more than 256 entries: a column has 32 threads, and blocks are many)
__global__ void __launch_bounds__(SCAN_THREADS, BATCH <= 2 ? 5 : BATCH == 4 ? 4 : 1)
state_scan_kernel(ScanParams p) {
  KVB_KERNEL_PROLOGUE(MODE == 0 ? KVB_TAG_GLA_SCAN : MODE == 1 ? KVB_TAG_DELTA_SCAN
                                                   : MODE == 2 ? KVB_TAG_LIGHTNING_SCAN : KVB_TAG_SSM_SCAN);
  extern __shared__ __align__(16) float smem[];
  constexpr int DP = DREG * RSPLIT;                 // rows covered (>= D; rows beyond D stay zero)
  constexpr int COLS = SCAN_THREADS / RSPLIT * CPT; // columns this block owns
  constexpr int NVEC = MODE == 0 ? 3 : 2;           // q, k (, a)
  constexpr int TOKEN = NVEC * DP + 4;              // floats a token holds in a stage; the last four: beta, gate
  constexpr int STAGE = BATCH * TOKEN;
  constexpr int VPT = (BATCH * COLS + SCAN_THREADS - 1) / SCAN_THREADS;
  constexpr int FPT = (BATCH * NVEC * (DP / 4) + SCAN_THREADS - 1) / SCAN_THREADS;   // 16-byte copies a thread, a stage
  constexpr int J = DREG / 4;
  constexpr int GROUP = BATCH < 8 ? BATCH : 8;      // tokens whose read-outs are summed over the threads together
  float* const vectors = smem;                      // [2][BATCH][TOKEN]
  float* const values = smem + 2 * STAGE;           // [2][BATCH][COLS][2]: every value twice, the halves of a pair

  const int req = blockIdx.x, h = blockIdx.y, tid = threadIdx.x;
  // neighbouring lanes hold the same rows of different columns: what they read of q and k is then the same word, which
  // the shared memory serves them at once
  constexpr int BESIDE = 32 / RSPLIT;               // columns (times CPT) a warp holds side by side
  const int part = (tid & 31) / BESIDE, c = ((tid >> 5) * BESIDE + (tid & 31) % BESIDE) * CPT;
  const int col = blockIdx.z * COLS + c;            // the first of this thread's columns
  const int begin = p.query_start[req], end = p.query_start[req + 1];
  const int D = p.D, V = p.V;
  const int kvh = h / p.kv_share;
  const TV* vg = (const TV*)p.v;

  // Thread `part` of a column holds the column's rows part * DREG .. part * DREG + DREG - 1 as J 16-byte pieces.
  // In shared memory a vector's piece n lies at place (n % J) * RSPLIT + n / J, so that for one j the parts of a
  // column read neighbouring pieces.
  float* const S_head = p.state + (size_t)p.state_slots[req] * p.state_stride + p.state_offset + (size_t)h * V * D;
  float4 held_state[CPT][J];                        // all of it on its way before any of it is looked at
#pragma unroll
  for (int cc = 0; cc < CPT; ++cc) {
    const float* S_column = S_head + (size_t)(col + cc < V ? col + cc : 0) * D;
#pragma unroll
    for (int j = 0; j < J; ++j) {
      const int row = part * DREG + 4 * j;
      float4 s4 = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      if (col + cc < V && row < D) {
        if (p.state16) {
          s4 = *reinterpret_cast<const float4*>(S_column + row);
        } else {
          s4.x = S_column[row];
          if (row + 1 < D) s4.y = S_column[row + 1];
          if (row + 2 < D) s4.z = S_column[row + 2];
          if (row + 3 < D) s4.w = S_column[row + 3];
        }
      }
      held_state[cc][j] = s4;
    }
  }
  ScanPair S[CPT][DREG / 2];
  auto place = [](int row) { return (((row >> 2) % J) * RSPLIT + (row >> 2) / J) * 4 + (row & 3); };
  if (D < DP)                                       // rows beyond D read zeros whatever the stage holds
    for (int e = tid; e < 2 * BATCH * NVEC * (DP - D); e += SCAN_THREADS) {
      const int slot = e / (DP - D), i = D + e % (DP - D);
      vectors[(slot / NVEC) * TOKEN + (slot % NVEC) * DP + place(i)] = 0.0f;
    }

  // Where this thread's 16-byte copies of a stage come from (for the stage that starts at token 0) and go to:
  // the same for every stage, so the divisions are taken once.
  const float* copy_from[FPT];
  int copy_to[FPT];
  const int pieces = D >> 2, per_token = NVEC * pieces;
  if (p.vec16) {
#pragma unroll
    for (int n = 0; n < FPT; ++n) {
      const int e = tid + n * SCAN_THREADS;
      const int tt = e / per_token, r = e - tt * per_token, vec = r / pieces, i = (r - vec * pieces) << 2;
      const float* base = vec == 0 ? p.q : vec == 1 ? p.k : p.a;
      copy_from[n] = base + (long long)tt * p.vec_token + (long long)(vec == 2 ? h : kvh) * D + i;
      copy_to[n] = tt * TOKEN + vec * DP + place(i);
    }
  }
  auto fetch = [&](int stage, int t0, int nb) {     // the vectors of tokens t0 .. t0 + nb - 1, asynchronously
    float* dst = vectors + stage * STAGE;
    if (p.vec16) {
      const long long shift = (long long)t0 * p.vec_token;
#pragma unroll
      for (int n = 0; n < FPT; ++n)
        if (tid + n * SCAN_THREADS < nb * per_token) scan_copy16(dst + copy_to[n], copy_from[n] + shift);
    } else {
      const int floats = NVEC * D;
      for (int e = tid; e < nb * floats; e += SCAN_THREADS) {
        const int tt = e / floats, r = e - tt * floats, vec = r / D, i = r - vec * D;
        const float* base = vec == 0 ? p.q : vec == 1 ? p.k : p.a;
        scan_copy4(dst + tt * TOKEN + vec * DP + place(i),
                   base + (long long)(t0 + tt) * p.vec_token + (long long)(vec == 2 ? h : kvh) * D + i);
      }
    }
    if (MODE == 1 || MODE == 3)
      for (int e = tid; e < 2 * nb; e += SCAN_THREADS) {
        const int tt = e >> 1;
        scan_copy4(dst + tt * TOKEN + NVEC * DP + (e & 1),
                   ((e & 1) ? p.gate : p.beta) + (size_t)(t0 + tt) * p.bg_stride + h);
      }
  };
  // This block's columns of v pass through registers, as they were stored: a conversion at the load would wait
  // for the load at the top of every stage.
  TV held[VPT];
  auto load_values = [&](int t0, int nb) {
#pragma unroll
    for (int j = 0; j < VPT; ++j) {
      const int e = tid + j * SCAN_THREADS, tt = e / COLS, cc = blockIdx.z * COLS + e % COLS;
      if (tt < nb && cc < V) held[j] = vg[(long long)(t0 + tt) * p.v_token + (long long)h * V + cc];
    }
  };
  auto store_values = [&](int stage, int nb) {
#pragma unroll
    for (int j = 0; j < VPT; ++j) {
      const int e = tid + j * SCAN_THREADS, tt = e / COLS, cc = blockIdx.z * COLS + e % COLS;
      const float v = (tt < nb && cc < V) ? to_float(held[j]) : 0.0f;
      if (e < BATCH * COLS) *reinterpret_cast<ScanPair*>(values + 2 * (stage * BATCH * COLS + e)) = scan_pair(v, v);
    }
  };
  const ScanPair head_decay = MODE == 2 ? scan_pair(p.a[h], p.a[h]) : 0;
  const float head_skip = MODE == 3 ? p.skip[h] : 0.0f;
  // The sums over the column's threads of the read-out are left to the caller, who takes them for all tokens of
  // a stage at once: those shuffles do not wait for one another, and the state's step does not wait for them.
  typedef ScanVectors<MODE, J, CPT> Vectors;
  auto take = [&](Vectors& n, const float* q, const float* vs) {
    const float* k = q + DP;
    if constexpr (CPT == 2) {
      const ulonglong2 v01 = *reinterpret_cast<const ulonglong2*>(vs);
      n.v[0] = v01.x; n.v[1] = v01.y;
    } else if constexpr (CPT == 4) {
      const ulonglong2 v01 = *reinterpret_cast<const ulonglong2*>(vs), v23 = *reinterpret_cast<const ulonglong2*>(vs + 4);
      n.v[0] = v01.x; n.v[1] = v01.y; n.v[2] = v23.x; n.v[3] = v23.y;
    } else {
#pragma unroll
      for (int cc = 0; cc < CPT; ++cc) n.v[cc] = *reinterpret_cast<const ScanPair*>(vs + 2 * cc);
    }
#pragma unroll
    for (int j = 0; j < J; ++j) {
      n.k4[j] = *reinterpret_cast<const ulonglong2*>(k + (j * RSPLIT + part) * 4);
      n.q4[j] = *reinterpret_cast<const ulonglong2*>(q + (j * RSPLIT + part) * 4);
      if (MODE == 0) n.a4[j] = *reinterpret_cast<const ulonglong2*>(k + DP + (j * RSPLIT + part) * 4);
    }
    if (MODE == 1 || MODE == 3) {
      const float2 two = *reinterpret_cast<const float2*>(q + NVEC * DP);
      n.first = two.x;
      n.second = two.y;
    }
  };
  auto token = [&](Vectors& n, float (&o_own)[CPT]) { scan_token<MODE, DREG, RSPLIT, CPT>(S, n, head_decay, o_own); };
  const bool out16 = CPT == 4 && (V & 3) == 0 && ((uintptr_t)p.out & 15) == 0;
  // the thread with part 0 writes its columns (and adds the token's own values, still in the stage, to them)
  auto write_out = [&](float* at, float (&sum)[CPT], const float* vs) {
    if (part != 0) return;
    if (MODE == 3)
#pragma unroll
      for (int cc = 0; cc < CPT; ++cc) sum[cc] = fmaf(head_skip, vs[2 * cc], sum[cc]);
    if (CPT == 4 && out16 && col < V) {
      *reinterpret_cast<float4*>(at) = make_float4(sum[0], sum[1], sum[2], sum[3]);
      return;
    }
#pragma unroll
    for (int cc = 0; cc < CPT; ++cc)
      if (col + cc < V) at[cc] = sum[cc];
  };

  if (begin < end) {
    fetch(0, begin, min(BATCH, end - begin));
    load_values(begin, min(BATCH, end - begin));
    store_values(0, min(BATCH, end - begin));
  }
  scan_copies_done();
  __syncthreads();
#pragma unroll
  for (int cc = 0; cc < CPT; ++cc)
#pragma unroll
    for (int j = 0; j < J; ++j) {
      S[cc][2 * j] = scan_pair(held_state[cc][j].x, held_state[cc][j].y);
      S[cc][2 * j + 1] = scan_pair(held_state[cc][j].z, held_state[cc][j].w);
    }
  int stage = 0;
  const size_t out_token = (size_t)p.heads * V;
  for (int t0 = begin; t0 < end; t0 += BATCH, stage ^= 1) {
    const int nb = min(BATCH, end - t0);
    const int next = t0 + BATCH, next_nb = min(BATCH, end - next);
    if (next < end) {
      fetch(stage ^ 1, next, next_nb);
      load_values(next, next_nb);
    }
    const float* st = vectors + stage * STAGE;
    const float* vs = values + 2 * (stage * BATCH * COLS + c);
    float* out_at = p.out + ((size_t)t0 * p.heads + h) * V + (col < V ? col : 0);
    if (BATCH > 2 && nb == BATCH) {                   // a full stage: nothing to ask between its tokens
      Vectors now;                                    // a token's vectors are read while the one in front is computed
      take(now, st, vs);
#pragma unroll
      for (int g = 0; g < BATCH; g += GROUP) {
        float sums[GROUP * CPT];                      // entry tt * CPT + cc
#pragma unroll
        for (int tt = 0; tt < GROUP; ++tt) {
          float own_part[CPT];
          Vectors next_one;
          if (g + tt + 1 < BATCH) take(next_one, st + (g + tt + 1) * TOKEN, vs + 2 * (g + tt + 1) * COLS);
          token(now, own_part);
          now = next_one;
#pragma unroll
          for (int cc = 0; cc < CPT; ++cc) sums[tt * CPT + cc] = own_part[cc];
        }
        constexpr int N = GROUP * CPT, LEFT = N > RSPLIT ? N / RSPLIT : 1;
        const int entry = scan_exchange<RSPLIT, N>(sums, part);
        if (part < N) {                               // with more threads than entries, several hold the same
#pragma unroll
          for (int i = 0; i < LEFT; ++i) {
            const int tt = g + (entry + i) / CPT, cc = (entry + i) % CPT;
            if (MODE == 3) sums[i] = fmaf(head_skip, vs[2 * (tt * COLS + cc)], sums[i]);
            if (col + cc < V) out_at[tt * out_token + cc] = sums[i];
          }
        }
      }
    } else {
      for (int tt = 0; tt < nb; ++tt) {
        float sum[CPT];
        Vectors now;
        take(now, st + tt * TOKEN, vs + 2 * tt * COLS);
        token(now, sum);
#pragma unroll
        for (int m = 1; m < RSPLIT; m <<= 1)
#pragma unroll
          for (int cc = 0; cc < CPT; ++cc) sum[cc] += __shfl_xor_sync(0xffffffffu, sum[cc], m * BESIDE);
        write_out(out_at + tt * out_token, sum, vs + 2 * tt * COLS);
      }
    }
    if (next < end) store_values(stage ^ 1, next_nb);
    scan_copies_done();
    __syncthreads();
  }
#pragma unroll
  for (int cc = 0; cc < CPT; ++cc) {
    if (col + cc >= V) continue;
    float* S_column = S_head + (size_t)(col + cc) * D;
#pragma unroll
    for (int j = 0; j < J; ++j) {
      const int row = part * DREG + 4 * j;
      if (row < D) {
        if (p.state16) {
          *reinterpret_cast<float4*>(S_column + row) =
              make_float4(scan_lo(S[cc][2 * j]), scan_hi(S[cc][2 * j]), scan_lo(S[cc][2 * j + 1]), scan_hi(S[cc][2 * j + 1]));
        } else {
          S_column[row] = scan_lo(S[cc][2 * j]);
          if (row + 1 < D) S_column[row + 1] = scan_hi(S[cc][2 * j]);
          if (row + 2 < D) S_column[row + 2] = scan_lo(S[cc][2 * j + 1]);
          if (row + 3 < D) S_column[row + 3] = scan_hi(S[cc][2 * j + 1]);
        }
      }
    }
  }
}

// The same scan of prompts whose vectors and values a tensor map can describe (keys of 16 to 256 entries, a multiple of four,
// rows and pointers on 16-byte boundaries): a warp of its own brings a stage's vectors, one box of [16 tokens] x [D] each, and values,
// [16 tokens] x [columns], through a ring of SCAN_DEPTH stages, and the warps that compute meet nobody.  Copies by those warps
// themselves cost more than their instructions, since whatever they load waits for the copies asked for in front of it.
#define SCAN_DEPTH 3
#define SCAN_STAGE 16                               // tokens a stage
#define SCAN_SPIN_LIMIT (1u << 20)

// WHOLE: the threads of a column hold no rows beyond D.
template <typename TV, int MODE, int DREG, int RSPLIT, int CPT>
struct ScanRing {
  static constexpr int DP = DREG * RSPLIT, COLS = SCAN_THREADS / RSPLIT * CPT, NVEC = MODE == 0 ? 3 : 2;
  static constexpr int VECTORS = NVEC * SCAN_STAGE * DP * 4, VALUES = SCAN_STAGE * COLS * (int)sizeof(TV);
  static constexpr int STAGE = VECTORS + VALUES + SCAN_STAGE * 8;         // beta and gate of a token, or dt and g
  static constexpr int BYTES = SCAN_DEPTH * STAGE + 128 + DREG * 4;       // barriers, zeros for threads without rows
  static_assert(STAGE % 128 == 0 && VALUES % 128 == 0, "a copy starts on a line");
};

struct ScanMaps { CUtensorMap q, k, a, v; };

template <typename TV, int MODE, int DREG, int RSPLIT, int CPT, bool WHOLE>
__global__ void __launch_bounds__(SCAN_THREADS + 32, 1)
state_scan_tma_kernel(const __grid_constant__ ScanMaps maps, const ScanParams p) {
  KVB_KERNEL_PROLOGUE(MODE == 0 ? KVB_TAG_GLA_SCAN : MODE == 1 ? KVB_TAG_DELTA_SCAN
                                                   : MODE == 2 ? KVB_TAG_LIGHTNING_SCAN : KVB_TAG_SSM_SCAN);
  using Ring = ScanRing<TV, MODE, DREG, RSPLIT, CPT>;
  constexpr int DP = Ring::DP, COLS = Ring::COLS, J = DREG / 4, GROUP = 8, BESIDE = 32 / RSPLIT;
  extern __shared__ __align__(128) unsigned char scan_dyn[];
  unsigned long long* full = reinterpret_cast<unsigned long long*>(scan_dyn + SCAN_DEPTH * Ring::STAGE);
  unsigned long long* empty = full + SCAN_DEPTH;
  float* const zeros = reinterpret_cast<float*>(scan_dyn + SCAN_DEPTH * Ring::STAGE + 128);
  const int pitch = WHOLE ? DP : p.D;               // a stage's vectors lie SCAN_STAGE * pitch apart
  const int req = blockIdx.x, h = blockIdx.y, warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int begin = p.query_start[req], end = p.query_start[req + 1];
  const int stages = (end - begin + SCAN_STAGE - 1) / SCAN_STAGE;
  if (threadIdx.x < DREG) zeros[threadIdx.x] = 0.0f;
  if (threadIdx.x == 0) {
    for (int s = 0; s < SCAN_DEPTH; ++s) {
      kvb_mbar_init(&full[s], MODE == 1 || MODE == 3 ? 33 : 1);
      kvb_mbar_init(&empty[s], SCAN_THREADS / 32);
    }
    kvb_mbar_init_fence();
  }
  __syncthreads();
  if (warp == SCAN_THREADS / 32) {
    // ================= vectors and values: the whole warp, one lane issues =================
    const unsigned leader = kvb_elect();
    const int kv_col = h / p.kv_share * p.D, v_col = h * p.V + blockIdx.z * COLS;
    int issued = 0;
    bool ok = true;
    for (int n = 0; n < stages; ++n) {
      const int s = n % SCAN_DEPTH, t0 = begin + n * SCAN_STAGE;
      if (n >= SCAN_DEPTH) ok = __all_sync(0xffffffffu, kvb_mbar_wait<SCAN_SPIN_LIMIT, 64>(&empty[s], ((n / SCAN_DEPTH) - 1) & 1));
      if (!ok) break;
      unsigned char* const at = scan_dyn + s * Ring::STAGE;
      if (leader) kvb_mbar_expect_tx(&full[s], Ring::NVEC * SCAN_STAGE * pitch * 4 + Ring::VALUES);
      kvb_tma_2d_by(at, &maps.q, kv_col, t0, &full[s], leader);
      kvb_tma_2d_by(at + SCAN_STAGE * pitch * 4, &maps.k, kv_col, t0, &full[s], leader);
      if (MODE == 0) kvb_tma_2d_by(at + 2 * SCAN_STAGE * pitch * 4, &maps.a, h * p.D, t0, &full[s], leader);
      kvb_tma_2d_by(at + Ring::VECTORS, &maps.v, v_col, t0, &full[s], leader);
      if (MODE == 1 || MODE == 3) {
        float* const two = reinterpret_cast<float*>(at + Ring::VECTORS + Ring::VALUES);
        const int t = t0 + (lane >> 1);
        if (t < end) scan_copy4(two + lane, ((lane & 1) ? p.gate : p.beta) + (size_t)t * p.bg_stride + h);
        asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];\n" ::"r"(kvb_smem(&full[s])) : "memory");
      }
      issued = n + 1;
    }
    if (!ok) {                                      // given up: let the copies in flight land before the block may exit
      if (lane == 0) atomicOr(p.status, KVB_STATUS_WAIT_TIMEOUT);
      for (int n = max(0, issued - SCAN_DEPTH); n < issued; ++n) kvb_mbar_wait<SCAN_SPIN_LIMIT, 64>(&full[n % SCAN_DEPTH], (n / SCAN_DEPTH) & 1);
      asm volatile("cp.async.wait_all;\n" ::: "memory");
    }
    return;
  }
  const int part = lane / BESIDE, c = (warp * BESIDE + lane % BESIDE) * CPT;
  const int col = blockIdx.z * COLS + c;            // the first of this thread's columns
  const int D = p.D, V = p.V;
  // thread `part` of a column holds the column's rows part * DREG .. part * DREG + DREG - 1
  float* const S_head = p.state + (size_t)p.state_slots[req] * p.state_stride + p.state_offset + (size_t)h * V * D;
  ScanPair S[CPT][DREG / 2];
#pragma unroll
  for (int cc = 0; cc < CPT; ++cc)
#pragma unroll
    for (int j = 0; j < J; ++j) {
      ulonglong2 s4 = make_ulonglong2(0, 0);
      if (col + cc < V && (WHOLE || part * DREG + 4 * j < D)) s4 = *reinterpret_cast<const ulonglong2*>(S_head + (size_t)(col + cc) * D + part * DREG + 4 * j);
      S[cc][2 * j] = s4.x;
      S[cc][2 * j + 1] = s4.y;
    }
  const ScanPair head_decay = MODE == 2 ? scan_pair(p.a[h], p.a[h]) : 0;
  const float head_skip = MODE == 3 ? p.skip[h] : 0.0f;
  typedef ScanVectors<MODE, J, CPT> Vectors;
  auto value = [&](const unsigned char* at, int tt, int cc) {
    return to_float(reinterpret_cast<const TV*>(at + Ring::VECTORS)[tt * COLS + c + cc]);
  };
  auto take = [&](Vectors& n, const unsigned char* at, int tt) {
#pragma unroll
    for (int j = 0; j < J; ++j) {
      const bool live = WHOLE || part * DREG + 4 * j < D;
      const float* q = live ? reinterpret_cast<const float*>(at) + tt * pitch + part * DREG + 4 * j : zeros;
      const int next = live ? SCAN_STAGE * pitch : 0;
      n.q4[j] = *reinterpret_cast<const ulonglong2*>(q);
      n.k4[j] = *reinterpret_cast<const ulonglong2*>(q + next);
      if (MODE == 0) n.a4[j] = *reinterpret_cast<const ulonglong2*>(q + 2 * next);
    }
    if constexpr (CPT == 4 && sizeof(TV) == 4) {
      const float4 v = *reinterpret_cast<const float4*>(reinterpret_cast<const TV*>(at + Ring::VECTORS) + tt * COLS + c);
      n.v[0] = scan_pair(v.x, v.x); n.v[1] = scan_pair(v.y, v.y); n.v[2] = scan_pair(v.z, v.z); n.v[3] = scan_pair(v.w, v.w);
    } else if constexpr (CPT == 2 && sizeof(TV) == 4) {
      const float2 v = *reinterpret_cast<const float2*>(reinterpret_cast<const TV*>(at + Ring::VECTORS) + tt * COLS + c);
      n.v[0] = scan_pair(v.x, v.x); n.v[1] = scan_pair(v.y, v.y);
    } else {
#pragma unroll
      for (int cc = 0; cc < CPT; ++cc) { const float v = value(at, tt, cc); n.v[cc] = scan_pair(v, v); }
    }
    if (MODE == 1 || MODE == 3) {
      const float2 two = reinterpret_cast<const float2*>(at + Ring::VECTORS + Ring::VALUES)[tt];
      n.first = two.x;
      n.second = two.y;
    }
  };
  const size_t out_token = (size_t)p.heads * V;
  bool ok = true;
  for (int n = 0; n < stages; ++n) {
    const int s = n % SCAN_DEPTH, t0 = begin + n * SCAN_STAGE, nb = min(SCAN_STAGE, end - t0);
    ok = __all_sync(0xffffffffu, kvb_mbar_wait<SCAN_SPIN_LIMIT, 64>(&full[s], (n / SCAN_DEPTH) & 1));
    if (!ok) break;
    const unsigned char* const at = scan_dyn + s * Ring::STAGE;
    float* const out_at = p.out + ((size_t)t0 * p.heads + h) * V + (col < V ? col : 0);
    if (nb == SCAN_STAGE) {
      Vectors now;                                  // a token's vectors are read while the one in front is computed
      take(now, at, 0);
#pragma unroll
      for (int g = 0; g < SCAN_STAGE; g += GROUP) {
        constexpr int N = GROUP * CPT, LEFT = N > RSPLIT ? N / RSPLIT : 1;
        float sums[N];                              // entry tt * CPT + cc
#pragma unroll
        for (int tt = 0; tt < GROUP; ++tt) {
          float own_part[CPT];
          Vectors next_one;
          if (g + tt + 1 < SCAN_STAGE) take(next_one, at, g + tt + 1);
          scan_token<MODE, DREG, RSPLIT, CPT>(S, now, head_decay, own_part);
          now = next_one;
#pragma unroll
          for (int cc = 0; cc < CPT; ++cc) sums[tt * CPT + cc] = own_part[cc];
        }
        const int entry = scan_exchange<RSPLIT, N>(sums, part);
        if (part < N) {                             // with more threads than entries, several hold the same
#pragma unroll
          for (int i = 0; i < LEFT; ++i) {
            const int tt = g + (entry + i) / CPT, cc = (entry + i) % CPT;
            if (MODE == 3) sums[i] = fmaf(head_skip, value(at, tt, cc), sums[i]);
            if (col + cc < V) out_at[tt * out_token + cc] = sums[i];
          }
        }
      }
    } else {
      for (int tt = 0; tt < nb; ++tt) {
        float sum[CPT];
        Vectors now;
        take(now, at, tt);
        scan_token<MODE, DREG, RSPLIT, CPT>(S, now, head_decay, sum);
#pragma unroll
        for (int m = 1; m < RSPLIT; m <<= 1)
#pragma unroll
          for (int cc = 0; cc < CPT; ++cc) sum[cc] += __shfl_xor_sync(0xffffffffu, sum[cc], m * BESIDE);
#pragma unroll
        for (int cc = 0; cc < CPT; ++cc) {
          if (MODE == 3) sum[cc] = fmaf(head_skip, value(at, tt, cc), sum[cc]);
          if (part == 0 && col + cc < V) out_at[tt * out_token + cc] = sum[cc];
        }
      }
    }
    __syncwarp();
    if (lane == 0) kvb_mbar_arrive(&empty[s]);
  }
  if (!ok) {
    if (lane == 0) atomicOr(p.status, KVB_STATUS_WAIT_TIMEOUT);
    return;
  }
#pragma unroll
  for (int cc = 0; cc < CPT; ++cc)
#pragma unroll
    for (int j = 0; j < J; ++j)
      if (col + cc < V && (WHOLE || part * DREG + 4 * j < D))
        *reinterpret_cast<ulonglong2*>(S_head + (size_t)(col + cc) * D + part * DREG + 4 * j) =
            make_ulonglong2(S[cc][2 * j], S[cc][2 * j + 1]);
}

// Rows of S a thread holds, how many neighbouring columns, and how many tokens a stage.  Sums over a column come out with the
// same bits whatever the choice, so it follows the launch.  A step of single tokens moves every state once and does little
// else: 8 rows of four columns, stages of two tokens (6 KB a block, so that many blocks share an SM).  A step with prompts in
// it takes as long as its fullest SM: blocks an SM times what a token costs a block, the least of the shapes below (the more
// columns a thread has, the more of them one load of q, k and the decays serves; the delta rule's chain passes through a sum
// over the column's threads, fewer with 16 rows).  Whole mixers at width 4,096 and 2,048 with keys of 128 (B200,
// microseconds, the scan the rest of them apart from 70 to 215): lightning, a prompt of 2,048, 4,096 columns: 8 x 4 400,
// 8 x 2 408, 8 x 1 569, 16 x 1 526 (455 with the copies made by the warps that compute, rows four at a time); retention, 1,024
// tokens, 2,048 columns: 150, 118, 150, 151 (165); state space, 4 prompts of 400, 16,384 columns: 281, 289, 386, 378 (335);
// gated linear, 1,024 tokens, 4,096 columns: 227, 257, 370, 351 (268); delta rule, prompts of 517, 460 and 403, 6,144 columns:
// 16 x 2 275, 8 x 4 301, 8 x 2 307, 16 x 1 308, 8 x 1 439 (318); one of 1,024, 2,048 columns: 247, 270, 209, 209, 313 (232);
// one of 500, 1,024 columns: 121, 135, 107, 105, 100 (137).
struct ScanShape { int rows, cols; bool brief; };
static long long scan_blocks(int D, long long heads_of_all, int V, int rows, int cols) {
  int rsplit = 1;
  while (rows * rsplit < D) rsplit *= 2;
  const int owned = SCAN_THREADS / rsplit * cols;
  return heads_of_all * ((V + owned - 1) / owned);
}
// tma: vectors and values may come by TMA.
static ScanShape scan_shape(int mode, int D, long long heads_of_all, int V, bool brief, bool tma) {
  const long long sms = kvb_sm_count() > 0 ? kvb_sm_count() : 148;
  int least = 8;                                      // 32 threads a column at most
  while (least * 32 < D) least *= 2;
  // tests run every choice on one input and compare the bits
  const char* rows_asked = getenv("KVCORE_SCAN_ROWS");
  const char* cols_asked = getenv("KVCORE_SCAN_COLS");
  const int r = rows_asked ? atoi(rows_asked) : 0, c = cols_asked ? atoi(cols_asked) : 0;
  if ((r == 8 || r == 16) && r >= least) return {r, c == 4 ? (r == 8 ? 4 : 2) : c == 2 ? 2 : 1, false};
  if (c == 4) return {least, least == 8 ? 4 : 2, brief && least == 8};
  if (c == 1) return {least, 1, false};
  // Single tokens with keys of 512, 16 heads of 512 values: 16 x 2 147 us, 16 x 1 167 (165 as four rows at a time); 64 heads 564 and 669 (636).
  if (brief) return least <= 8 ? ScanShape{8, 4, true} : ScanShape{16, 2, false};
  if (least > 8) return {least, 1, false};
  // Keys that leave threads without rows come by TMA in the shape 8 x 2 alone.  Beyond 128 entries a stage of them takes the room
  // of 256, one block fits an SM (three vectors a token) or two, and with more blocks than that 8 x 4 by copies is sooner done.
  // 64 heads of 128 values, 4 prompts of 100, keys of 192: gated linear 8 x 2 388, 8 x 4 271, lightning 249 and 214; 4 heads, one
  // prompt of 300: 44 and 69, 36 and 56; keys of 96 with 96 values, 64 heads, 32 prompts of 33: 286 and 302, 214 and 250.
  // (Values that no map describes leave the choice to the costs below: gated linear, keys and values of 100, 64 heads, 32 prompts of
  // 33: 8 x 4 by copies 388, 8 x 2 by copies 505.)
  const bool spare = tma && (D & (D - 1)) != 0;
  if (spare && mode != 1)
    return D <= 128 || scan_blocks(D, heads_of_all, V, 8, 2) <= (mode == 0 ? 1 : 2) * sms ? ScanShape{8, 2, false} : ScanShape{8, 4, false};
  // Delta rule, keys of 256 (two blocks of 16 x 2 an SM by their stages): 16 heads of 128 values, 32 prompts of 33: 8 x 4 by copies
  // 232, 16 x 2 260; one prompt of 300: 92 and 74.
  if (mode == 1 && D == 256 && scan_blocks(D, heads_of_all, V, 16, 2) > 3 * sms) return {8, 4, false};
  struct { int rows, cols; double cost; } const fixed[] = {{8, 1, 0.5}, {8, 2, 0.6}, {8, 4, 1.0}}, delta[] = {{8, 1, 0.72}, {8, 2, 0.79}, {16, 2, 1.0}};
  ScanShape best = {8, 1, false};
  double least_cost = 0.0;
  for (const auto& o : mode == 1 ? delta : fixed) {
    if (spare && o.cols == 1) continue;               // 16 heads of 128 values, 32 prompts of 33, keys of 192: 8 x 1 628, 8 x 2 382, 16 x 2 210
    const double cost = (double)((scan_blocks(D, heads_of_all, V, o.rows, o.cols) + sms - 1) / sms) * o.cost;
    if (least_cost > 0.0 && cost >= least_cost) continue;
    least_cost = cost;
    best = {o.rows, o.cols, false};
  }
  return best;
}

// Whether tensor maps describe the vectors and values of a launch, but for the width of its blocks, and the maps.
static bool scan_by_tma(const ScanParams& p, size_t e, long long tokens) {
  return p.D % 4 == 0 && p.D <= 256 && p.D >= 16 && p.vec16 && p.state16 && tokens < (1ll << 31) && p.V * e % 16 == 0 &&
         (size_t)p.v_token * e % 16 == 0 && aligned16(p.v) && (size_t)p.vec_token * 4 % 16 == 0 &&
         (long long)p.heads * p.V < (1ll << 31) && (long long)p.heads * p.D < (1ll << 31);
}
template <typename TV>
static bool scan_maps(ScanMaps* maps, const ScanParams& p, int mode, int cols, long long tokens) {
  const size_t e = sizeof(TV);
  if (!scan_by_tma(p, e, tokens) || cols > 256 || cols * e % 16) return false;
  KvbEncodeTiledFn encode = kvb_encode_tiled_fn();
  if (encode == nullptr) return false;
  const cuuint32_t elem[2] = {1, 1};
  auto make = [&](CUtensorMap* map, CUtensorMapDataType type, const void* base, long long width, long long stride_bytes, int box_width) {
    const cuuint64_t dims[2] = {(cuuint64_t)width, (cuuint64_t)tokens};
    const cuuint64_t strides[1] = {(cuuint64_t)stride_bytes};
    const cuuint32_t box[2] = {(cuuint32_t)box_width, SCAN_STAGE};
    return encode(map, type, 2, const_cast<void*>(base), dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
                  CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
  };
  const CUtensorMapDataType f32 = CU_TENSOR_MAP_DATA_TYPE_FLOAT32;
  const long long kv_width = (long long)(p.heads / p.kv_share) * p.D;
  return make(&maps->q, f32, p.q, kv_width, p.vec_token * 4, p.D) && make(&maps->k, f32, p.k, kv_width, p.vec_token * 4, p.D) &&
         (mode != 0 || make(&maps->a, f32, p.a, (long long)p.heads * p.D, p.vec_token * 4, p.D)) &&
         make(&maps->v, e == 4 ? f32 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, p.v, (long long)p.heads * p.V, p.v_token * (long long)e, cols);
}

template <typename TV, int MODE>
static int launch_state_scan(const ScanParams& p_in, int num_reqs, long long tokens, cudaStream_t stream) {
  ScanParams p = p_in;
  KVB_REQUIRE(p.D <= 512, "state_scan: keys wider than 512 entries");
  p.vec16 = (p.D % 4 == 0 && p.vec_token % 4 == 0 &&
             ((uintptr_t)p.q | (uintptr_t)p.k | (MODE == 2 ? 0 : (uintptr_t)p.a)) % 16 == 0) ? 1 : 0;
  p.state16 = (p.D % 4 == 0 && p.state_stride % 4 == 0 && p.state_offset % 4 == 0 && (uintptr_t)p.state % 16 == 0) ? 1 : 0;
  const ScanShape shape = scan_shape(MODE, p.D, (long long)num_reqs * p.heads, p.V, tokens <= 2LL * num_reqs,
                                     scan_by_tma(p, sizeof(TV), tokens));
  const int dreg = shape.rows, cpt = shape.cols;
  int rsplit = 1;
  while (dreg * rsplit < p.D) rsplit *= 2;
  const int cols = SCAN_THREADS / rsplit * cpt;
  const dim3 grid(num_reqs, p.heads, (p.V + cols - 1) / cols), block(SCAN_THREADS);
  cudaError_t err = cudaErrorInvalidValue;
  // A launch with prompts in it lasts as long as its fullest SM.  Its blocks may come in while the kernel in front
  // still holds some SMs (dependent launch) and would then crowd on the others: each asks for so much shared memory
  // that no SM holds more of them than its share.
  const long long sms = kvb_sm_count() > 0 ? kvb_sm_count() : 148;
  const long long blocks = (long long)grid.x * grid.y * grid.z, share = (blocks + sms - 1) / sms;
  const size_t alone = !shape.brief && share <= 8 ? SCAN_SM_BYTES / (size_t)(share + 1) : 0;
#define SCAN_CASE(DR, RS, CP, BRIEF)                                                                          \
  if (dreg == DR && rsplit == RS && cpt == CP && shape.brief == BRIEF) {                                      \
    constexpr int B = BRIEF ? 2 : DR * RS <= 128 ? 16 : 2048 / (DR * RS);                                     \
    constexpr size_t need = 2 * (size_t)B * ((MODE == 0 ? 3 : 2) * DR * RS + 4 + 2 * (SCAN_THREADS / RS * CP)) * sizeof(float); \
    const size_t smem = need < alone ? alone : need;                                                          \
    if (smem > 48 * 1024)           /* the most that any launch asks for: another thread's may be in between */ \
      KVB_CHECK_CUDA(cudaFuncSetAttribute(state_scan_kernel<TV, MODE, DR, RS, CP, B>, cudaFuncAttributeMaxDynamicSharedMemorySize, \
                                          (int)(need < SCAN_SM_BYTES / 2 ? SCAN_SM_BYTES / 2 : need)));       \
    err = kvb_launch((state_scan_kernel<TV, MODE, DR, RS, CP, B>), grid, block, smem, stream, true, p);       \
  }
#define SCAN_ROWS(DR, CP, BRIEF)                                                                              \
  SCAN_CASE(DR, 1, CP, BRIEF) SCAN_CASE(DR, 2, CP, BRIEF) SCAN_CASE(DR, 4, CP, BRIEF) SCAN_CASE(DR, 8, CP, BRIEF) \
  SCAN_CASE(DR, 16, CP, BRIEF) SCAN_CASE(DR, 32, CP, BRIEF)
  ScanMaps maps = {};
  p.status = kvb_status_word();
  KVB_REQUIRE(p.status != nullptr, "state_scan: no status word");
  if (!shape.brief && scan_maps<TV>(&maps, p, MODE, cols, tokens)) {
#define SCAN_TMA(DR, RS, CP, WHOLE)                                                                           \
    if (dreg == DR && rsplit == RS && cpt == CP && (p.D == DR * RS) == WHOLE) {                               \
      using Ring = ScanRing<TV, MODE, DR, RS, CP>;                                                            \
      const size_t smem = Ring::BYTES < alone ? alone : Ring::BYTES;                                          \
      KVB_CHECK_CUDA(cudaFuncSetAttribute(state_scan_tma_kernel<TV, MODE, DR, RS, CP, WHOLE>, cudaFuncAttributeMaxDynamicSharedMemorySize, \
                                          Ring::BYTES < SCAN_SM_BYTES / 2 ? SCAN_SM_BYTES / 2 : Ring::BYTES)); \
      KVB_CHECK_CUDA(kvb_launch((state_scan_tma_kernel<TV, MODE, DR, RS, CP, WHOLE>), grid, dim3(SCAN_THREADS + 32), smem, stream, true, \
                                maps, p));                                                                    \
      KVB_CHECK_LAUNCH();                                                                                     \
      return 0;                                                                                               \
    }
#define SCAN_TMA_KEYS(DR, CP) SCAN_TMA(DR, 16 / DR, CP, true) SCAN_TMA(DR, 32 / DR, CP, true) SCAN_TMA(DR, 64 / DR, CP, true) \
    SCAN_TMA(DR, 128 / DR, CP, true) SCAN_TMA(DR, 256 / DR, CP, true)
    SCAN_TMA_KEYS(8, 1) SCAN_TMA_KEYS(8, 2)
    if constexpr (MODE == 1) { SCAN_TMA_KEYS(16, 2) } else { SCAN_TMA_KEYS(8, 4) }
    SCAN_TMA(8, 4, 2, false) SCAN_TMA(8, 8, 2, false) SCAN_TMA(8, 16, 2, false) SCAN_TMA(8, 32, 2, false)
#undef SCAN_TMA_KEYS
#undef SCAN_TMA
  }
  SCAN_ROWS(8, 1, false) SCAN_ROWS(8, 2, false) SCAN_ROWS(8, 4, false) SCAN_ROWS(16, 1, false) SCAN_ROWS(16, 2, false)
  SCAN_ROWS(16, 1, true) SCAN_ROWS(8, 4, true)
#undef SCAN_ROWS
#undef SCAN_CASE
  KVB_CHECK_CUDA(err);
  KVB_CHECK_LAUNCH();
  return 0;
}
