// The gated delta rule of delta_rule.cu over long portions, by chunks of 64 tokens:
//
//     S <- g S;   u = beta (v - S^T k);   S <- S + k u^T;   o = S^T q.
//
// With G_t = g_1 .. g_t inside a chunk that found the state S0, and D_ts = g_(s+1) .. g_t, the writes of a chunk solve
//
//     (I + L) U = diag(beta) (V - diag(G) K S0),     L_ts = beta_t D_ts (k_s . k_t) for s < t,
//
// so U = X - Y S0 with  (I + L) X = diag(beta) V  and  (I + L) Y = diag(beta G) K,  which need no state (the chunkwise form of
// the delta rule: S. Yang et al., "Parallelizing Linear Transformers with the Delta Rule over Sequence Length", 2024; with decays:
// "Gated Delta Networks", 2024):
//
//   delta_solve    X and Y of all chunks and heads at once, by forward substitution, a thread per column.
//   delta_chain    the one dependent chain: per request, head and slice of value columns, chunk after chunk,
//                  U = X - Y S,  S <- G_end S + sum_s D_end,s k_s u_s^T;  it leaves every chunk's U and start state.
//   delta_outputs  o_t = G_t S0^T q_t + sum_{s<=t} D_ts (k_s . q_t) u_s, all chunks and heads at once.
//
// D and G are running products of decays, never quotients; everything is 32-bit (two FMAs per instruction).  A token's sums
// depend on where it stands in its chunk, and chunks count from the request's first token of the step.
// Bound by 32-bit FMAs (150 thousand per token and head, 98 by the walk, which a chain of 2048 steps keeps from them) and by the
// chain's meetings.  16 heads of 128 x 128, 2048 tokens, with a portion that starts from a state: solve 44 us, chain 142, outputs
// 64, together 259 (the walk 538); 512 tokens 83 (198); 32 heads 2048 tokens 419 (550).  Errors against 64 bits, of the outputs'
// and the state's length: 1.1e-7 and 5.3e-8 (the walk 9.3e-8 and 5.4e-8).
#include "common.cuh"

#define CHUNK 64
#define PIECE 16
#define PIECES (CHUNK / PIECE)
#define DC_D 128     // channels and value columns a head may have (zeros beyond its own)
#define DC_LD 132
#define DC_LDL 68
#define DC_THREADS 256
#define DC_CS 16       // value columns of a block of the chain

struct DeltaChunkParams {
  const float* q;      // [N, G, dk]
  const float* k;      // [N, G, dk]
  const float* v;      // [N, H, dv]
  const float* beta;   // [N, H]
  const float* decay;  // [N, H]
  const int* chunks;   // [n, 3]: request, first token row, end row; a request's chunks in order
  const int* requests; // [m, 3]: request, its first chunk, its chunks
  const int* slot_ids;
  float* state;        // [slots, H, dk, dv]
  float* o;            // [N, H, dv]
  float* X;            // [n, H, CHUNK, dv]: X, then U
  float* Y;            // [n, H, CHUNK, dk]
  float* S0;           // [n, H, dk, dv]
  float* ends;         // [n, H, CHUNK]: D_end,t
  float* wholes;       // [n, H]: G_end
  int G, H, dk, dv;
};

typedef unsigned long long u64;
__device__ __forceinline__ u64 dc_fma2(u64 a, u64 b, u64 c) {
  u64 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ u64 dc_add2(u64 a, u64 b) {
  u64 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ u64 dc_pair(float x, float y) { return (u64)__float_as_uint(x) | ((u64)__float_as_uint(y) << 32); }
__device__ __forceinline__ u64 dc_twice(float x) { return dc_pair(x, x); }
__device__ __forceinline__ float dc_low(u64 p) { return __uint_as_float((unsigned)p); }
__device__ __forceinline__ float dc_high(u64 p) { return __uint_as_float((unsigned)(p >> 32)); }
__device__ __forceinline__ void dc_copy16(float* dst, const float* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void dc_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void dc_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// rows x cols of a matrix with rows `ld` apart into shared memory, zeros from `cnt` rows and
// `size` columns on.  Sizes are multiples of 4.
__device__ __forceinline__ void dc_load(float* dst, int ld_dst, const float* src, size_t ld, int rows, int cols, int cnt, int size) {
#pragma unroll 4
  for (int idx = threadIdx.x; idx < rows * (cols / 4); idx += DC_THREADS) {
    const int t = idx / (cols / 4), c = idx % (cols / 4) * 4;
    if (t < cnt && c < size) dc_copy16(dst + t * ld_dst + c, src + (size_t)t * ld + c);
    else *reinterpret_cast<float4*>(dst + t * ld_dst + c) = make_float4(0.f, 0.f, 0.f, 0.f);
  }
}

// The chunk's decays g[CHUNK] (one from the chunk's end on) in, per token the products from its piece's start (with its own)
// and to its piece's end (without its own), and the pieces' products.  Threads 0 .. 7 work; the caller synchronises.
__device__ __forceinline__ void dc_products(const float* g, float* from, float* to, float* piece) {
  const int p = threadIdx.x & 3;
  if (threadIdx.x < 4) {
    float x = 1.f;
    for (int t = p * PIECE; t < (p + 1) * PIECE; ++t) {
      x *= g[t];
      from[t] = x;
    }
    piece[p] = x;
  } else if (threadIdx.x < 8) {
    float x = 1.f;
    for (int t = (p + 1) * PIECE - 1; t >= p * PIECE; --t) {
      to[t] = x;
      x *= g[t];
    }
  }
}
// D_ts for s <= t
__device__ __forceinline__ float dc_between(const float* g, const float* from, const float* to, const float* piece, int t, int s) {
  const int p = t / PIECE, b = s / PIECE;
  if (p == b) {
    float x = 1.f;
    for (int r = s + 1; r <= t; ++r) x *= g[r];
    return x;
  }
  float x = to[s];
  for (int r = b + 1; r < p; ++r) x *= piece[r];
  return x * from[t];
}
__device__ __forceinline__ float dc_from_start(const float* from, const float* piece, int t) {
  float x = from[t];
  for (int r = 0; r < t / PIECE; ++r) x *= piece[r];
  return x;
}
__device__ __forceinline__ float dc_to_end(const float* to, const float* piece, int s) {
  float x = to[s];
  for (int r = s / PIECE + 1; r < PIECES; ++r) x *= piece[r];
  return x;
}

// x_t . y_s by pieces of 16 x 16 on and below the diagonal, rows of shared memory: thread (t, s) of each piece.  Eight short sums
// (32 channels, even and odd) per product: half the error of two long ones.
__device__ __forceinline__ void dc_piece_products(const float* X, const float* Y, int tl, int sl, float (&out)[PIECES][PIECES]) {
  u64 total[PIECES][PIECES];
#pragma unroll
  for (int p = 0; p < PIECES; ++p)
#pragma unroll
    for (int b = 0; b < PIECES; ++b) total[p][b] = 0ull;
#pragma unroll 1
  for (int c0 = 0; c0 < DC_D; c0 += 32) {
    u64 sum[PIECES][PIECES];
#pragma unroll
    for (int p = 0; p < PIECES; ++p)
#pragma unroll
      for (int b = 0; b < PIECES; ++b) sum[p][b] = 0ull;
#pragma unroll 2
    for (int c = c0; c < c0 + 32; c += 4) {
      ulonglong2 y[PIECES];
#pragma unroll
      for (int b = 0; b < PIECES; ++b) y[b] = *reinterpret_cast<const ulonglong2*>(Y + (b * PIECE + sl) * DC_LD + c);
#pragma unroll
      for (int p = 0; p < PIECES; ++p) {
        const ulonglong2 x = *reinterpret_cast<const ulonglong2*>(X + (p * PIECE + tl) * DC_LD + c);
#pragma unroll
        for (int b = 0; b <= p; ++b) sum[p][b] = dc_fma2(x.y, y[b].y, dc_fma2(x.x, y[b].x, sum[p][b]));
      }
    }
#pragma unroll
    for (int p = 0; p < PIECES; ++p)
#pragma unroll
      for (int b = 0; b <= p; ++b) total[p][b] = dc_add2(total[p][b], sum[p][b]);
  }
#pragma unroll
  for (int p = 0; p < PIECES; ++p)
#pragma unroll
    for (int b = 0; b <= p; ++b) out[p][b] = dc_low(total[p][b]) + dc_high(total[p][b]);
}

__global__ void __launch_bounds__(DC_THREADS, 2) delta_solve_kernel(const __grid_constant__ DeltaChunkParams P) {
  JLX_TL(TL_OTHER);
  extern __shared__ __align__(16) float smem[];
  float* K = smem;                    // [CHUNK][DC_LD]
  float* V = K + CHUNK * DC_LD;       // [CHUNK][DC_LD]
  float* L = V + CHUNK * DC_LD;       // [s][t]: L_ts at s * DC_LDL + t
  __shared__ float g[CHUNK], beta[CHUNK], beta_from_start[CHUNK], from[CHUNK], to[CHUNK], piece[PIECES];
  const int chunk = blockIdx.x, h = blockIdx.y, tid = threadIdx.x;
  const int n0 = P.chunks[3 * chunk + 1], cnt = P.chunks[3 * chunk + 2] - n0;
  const int kh = h / (P.H / P.G);
  dc_load(K, DC_LD, P.k + ((size_t)n0 * P.G + kh) * P.dk, (size_t)P.G * P.dk, CHUNK, DC_D, cnt, P.dk);
  dc_commit();
  dc_load(V, DC_LD, P.v + ((size_t)n0 * P.H + h) * P.dv, (size_t)P.H * P.dv, CHUNK, DC_D, cnt, P.dv);
  dc_commit();
  if (tid < CHUNK) {
    g[tid] = tid < cnt ? P.decay[(size_t)(n0 + tid) * P.H + h] : 1.f;
    beta[tid] = tid < cnt ? P.beta[(size_t)(n0 + tid) * P.H + h] : 0.f;
  }
  dc_wait<1>();
  __syncthreads();
  dc_products(g, from, to, piece);
  const int sl = tid & 15, tl = tid >> 4;
  float sum[PIECES][PIECES];
  dc_piece_products(K, K, tl, sl, sum);
  __syncthreads();  // the products of decays are there
  if (tid < CHUNK) {
    P.ends[((size_t)chunk * P.H + h) * CHUNK + tid] = dc_to_end(to, piece, tid);
    beta_from_start[tid] = beta[tid] * dc_from_start(from, piece, tid);
  }
  if (tid == CHUNK) P.wholes[(size_t)chunk * P.H + h] = piece[0] * piece[1] * piece[2] * piece[3];
#pragma unroll
  for (int p = 0; p < PIECES; ++p)
#pragma unroll
    for (int b = 0; b <= p; ++b) {
      const int t = p * PIECE + tl, s = b * PIECE + sl;
      L[s * DC_LDL + t] = s < t ? beta[t] * dc_between(g, from, to, piece, t, s) * sum[p][b] : 0.f;
    }
  dc_wait<0>();
  __syncthreads();
  // columns 0 .. 127: of X (value columns); 128 .. 255: of Y (channels).  A thread solves its column: what the rows before take
  // off each row is summed in its registers by itself (small numbers among themselves), and the right side joins at the row's turn.
  const bool is_y = tid >= DC_D;
  const int c = tid & (DC_D - 1), size = is_y ? P.dk : P.dv;
  if (c >= size) return;
  float* out = (is_y ? P.Y + ((size_t)chunk * P.H + h) * CHUNK * P.dk : P.X + ((size_t)chunk * P.H + h) * CHUNK * P.dv) + c;
  const float* right = (is_y ? K : V) + c;
  const float* scale = is_y ? beta_from_start : beta;
  u64 acc[CHUNK / 2];
#pragma unroll
  for (int i = 0; i < CHUNK / 2; ++i) acc[i] = 0ull;
#pragma unroll
  for (int s = 0; s < CHUNK; ++s) {  // row s is done, and goes off the rows behind it
    const float x = fmaf(scale[s], right[s * DC_LD], (s & 1) ? dc_high(acc[s / 2]) : dc_low(acc[s / 2]));
    out[(size_t)s * size] = x;
    const u64 xx = dc_twice(-x);
    const float* l = L + s * DC_LDL;
    if ((s & 3) == 0) acc[s / 2] = dc_fma2(xx, *reinterpret_cast<const u64*>(l + s), acc[s / 2]);  // (L_ss is zero)
    if ((s & 3) <= 1) acc[(s & ~3) / 2 + 1] = dc_fma2(xx, *reinterpret_cast<const u64*>(l + (s & ~3) + 2), acc[(s & ~3) / 2 + 1]);
    if ((s & 3) == 2) acc[s / 2] = dc_fma2(xx, *reinterpret_cast<const u64*>(l + s), acc[s / 2]);
#pragma unroll
    for (int t = (s & ~3) + 4; t < CHUNK; t += 4) {
      const ulonglong2 y = *reinterpret_cast<const ulonglong2*>(l + t);
      acc[t / 2] = dc_fma2(xx, y.x, acc[t / 2]);
      acc[t / 2 + 1] = dc_fma2(xx, y.y, acc[t / 2 + 1]);
    }
  }
}

// 16 value columns and 256 threads per block, two blocks a multiprocessor.  Two products per chunk, each cut over its sum into four
// groups of threads whose parts meet in shared memory; a thread has 4 x 4 (Y S) or 8 x 4 (k u^T) outputs.  One stage of rows: the
// next chunk's Y and X arrive during the second product, its keys during the next first one.  (Two stages and one block a
// multiprocessor: 132 us for 142 above, but 8 requests of 256 tokens 255 us for 224.)
__global__ void __launch_bounds__(DC_THREADS, 2) delta_chain_kernel(const __grid_constant__ DeltaChunkParams P) {
  JLX_TL(TL_OTHER);
  constexpr int CS = DC_CS, JG = CS / 4, KG = 4;  // columns, column groups, sum groups
  extern __shared__ __align__(16) float smem[];
  float* Y = smem;                    // [CHUNK][DC_LD]
  float* K = Y + CHUNK * DC_LD;       // [CHUNK][DC_LD]
  float* Xs = K + CHUNK * DC_LD;      // two chunks' [CHUNK][CS]
  float* S = Xs + 2 * CHUNK * CS;     // [DC_D][CS]
  float* U = S + DC_D * CS;           // [CHUNK][CS]: u_s times D_end,s
  float* part = U + CHUNK * CS;       // [KG - 1][DC_D][CS]: the parts of all groups but the first
  __shared__ float ends[2][CHUNK], wholes[2];
  const int tid = threadIdx.x, h = blockIdx.y, j0 = blockIdx.z * CS, kh = h / (P.H / P.G);
  const int r = P.requests[3 * blockIdx.x], first = P.requests[3 * blockIdx.x + 1], count = P.requests[3 * blockIdx.x + 2];
  const int cols = min(CS, P.dv - j0);
  float* home = P.state + ((size_t)P.slot_ids[r] * P.H + h) * P.dk * P.dv + j0;
  for (int idx = tid; idx < DC_D * CS; idx += DC_THREADS) {
    const int c = idx / CS, j = idx % CS;
    S[idx] = c < P.dk && j < cols ? home[(size_t)c * P.dv + j] : 0.f;
  }
  auto fetch_solution = [&](int i) {  // always a group of copies, maybe an empty one
    if (i < count) {
      const size_t at = (size_t)(first + i) * P.H + h;
      dc_load(Y, DC_LD, P.Y + at * CHUNK * P.dk, P.dk, CHUNK, DC_D, CHUNK, P.dk);
      dc_load(Xs + (i & 1) * CHUNK * CS, CS, P.X + at * CHUNK * P.dv + j0, P.dv, CHUNK, CS, CHUNK, cols);
      if (tid < CHUNK) ends[i & 1][tid] = P.ends[at * CHUNK + tid];
      if (tid == CHUNK) wholes[i & 1] = P.wholes[at];
    }
    dc_commit();
  };
  auto fetch_keys = [&](int i) {
    if (i < count) {
      const int chunk = first + i, n0 = P.chunks[3 * chunk + 1], cnt = P.chunks[3 * chunk + 2] - n0;
      dc_load(K, DC_LD, P.k + ((size_t)n0 * P.G + kh) * P.dk, (size_t)P.G * P.dk, CHUNK, DC_D, cnt, P.dk);
    }
    dc_commit();
  };
  fetch_solution(0);
  fetch_keys(0);
  const int jg = tid % JG, rg = tid / JG % 16, kg = tid / (JG * 16);
#pragma unroll 1
  for (int i = 0; i < count; ++i) {
    dc_wait<1>();
    __syncthreads();  // this chunk's Y and X and the state that it finds are there
    const float whole = wholes[i & 1];
    const float* X = Xs + (i & 1) * CHUNK * CS;
    const size_t at = (size_t)(first + i) * P.H + h;
    {
      float* s0 = P.S0 + at * P.dk * P.dv + j0;
      for (int idx = tid; idx < DC_D * (CS / 4); idx += DC_THREADS) {
        const int c = idx / (CS / 4), j = idx % (CS / 4) * 4;
        if (c < P.dk && j < cols) *reinterpret_cast<float4*>(s0 + (size_t)c * P.dv + j) = *reinterpret_cast<const float4*>(S + c * CS + j);
      }
    }
    {  // Y S: rows rg + 16 a, columns 4 jg .., channels of the thread's group
      u64 acc[4][2];
#pragma unroll
      for (int a = 0; a < 4; ++a) acc[a][0] = acc[a][1] = 0ull;
#pragma unroll 4
      for (int c = kg * (DC_D / KG); c < (kg + 1) * (DC_D / KG); c += 4) {
        float4 y[4];
#pragma unroll
        for (int a = 0; a < 4; ++a) y[a] = *reinterpret_cast<const float4*>(Y + (rg + 16 * a) * DC_LD + c);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const ulonglong2 s = *reinterpret_cast<const ulonglong2*>(S + (c + e) * CS + 4 * jg);
#pragma unroll
          for (int a = 0; a < 4; ++a) {
            const u64 x = dc_twice(e == 0 ? y[a].x : (e == 1 ? y[a].y : (e == 2 ? y[a].z : y[a].w)));
            acc[a][0] = dc_fma2(x, s.x, acc[a][0]);
            acc[a][1] = dc_fma2(x, s.y, acc[a][1]);
          }
        }
      }
      if (kg > 0)
#pragma unroll
        for (int a = 0; a < 4; ++a)
          *reinterpret_cast<ulonglong2*>(part + ((kg - 1) * CHUNK + rg + 16 * a) * CS + 4 * jg) = make_ulonglong2(acc[a][0], acc[a][1]);
      __syncthreads();
      fetch_solution(i + 1);  // Y is read; X goes into the other half
      if (kg == 0) {  // the first group adds the others' parts to its own
#pragma unroll
        for (int a = 0; a < 4; ++a) {
          const int t = rg + 16 * a, idx = t * CS + 4 * jg;
          float4 s = make_float4(dc_low(acc[a][0]), dc_high(acc[a][0]), dc_low(acc[a][1]), dc_high(acc[a][1]));
#pragma unroll
          for (int z = 0; z < KG - 1; ++z) {
            const float4 p = *reinterpret_cast<const float4*>(part + z * CHUNK * CS + idx);
            s = make_float4(s.x + p.x, s.y + p.y, s.z + p.z, s.w + p.w);
          }
          const float4 x = *reinterpret_cast<const float4*>(X + idx);
          const float4 u = make_float4(x.x - s.x, x.y - s.y, x.z - s.z, x.w - s.w);
          const float e = ends[i & 1][t];
          *reinterpret_cast<float4*>(U + idx) = make_float4(u.x * e, u.y * e, u.z * e, u.w * e);
          if (4 * jg < cols) *reinterpret_cast<float4*>(P.X + at * CHUNK * P.dv + (size_t)t * P.dv + j0 + 4 * jg) = u;
        }
      }
    }
    dc_wait<1>();
    __syncthreads();  // the keys and u are there
    {  // k u^T: channels 4 rg .. and 64 + 4 rg .., columns 4 jg .., tokens of the thread's group
      u64 acc[8][2];
#pragma unroll
      for (int a = 0; a < 8; ++a) acc[a][0] = acc[a][1] = 0ull;
#pragma unroll 8
      for (int t = kg * (CHUNK / KG); t < (kg + 1) * (CHUNK / KG); ++t) {
        const float4 k0 = *reinterpret_cast<const float4*>(K + t * DC_LD + 4 * rg), k1 = *reinterpret_cast<const float4*>(K + t * DC_LD + 64 + 4 * rg);
        const ulonglong2 u = *reinterpret_cast<const ulonglong2*>(U + t * CS + 4 * jg);
        const float k[8] = {k0.x, k0.y, k0.z, k0.w, k1.x, k1.y, k1.z, k1.w};
#pragma unroll
        for (int a = 0; a < 8; ++a) {
          const u64 x = dc_twice(k[a]);
          acc[a][0] = dc_fma2(x, u.x, acc[a][0]);
          acc[a][1] = dc_fma2(x, u.y, acc[a][1]);
        }
      }
      if (kg > 0)
#pragma unroll
        for (int a = 0; a < 8; ++a)
          *reinterpret_cast<ulonglong2*>(part + ((kg - 1) * DC_D + (a < 4 ? 0 : 64) + 4 * rg + (a & 3)) * CS + 4 * jg) = make_ulonglong2(acc[a][0], acc[a][1]);
      __syncthreads();
      fetch_keys(i + 1);  // the keys are read
      if (kg == 0) {
#pragma unroll
        for (int a = 0; a < 8; ++a) {
          const int idx = ((a < 4 ? 0 : 64) + 4 * rg + (a & 3)) * CS + 4 * jg;
          float4 s = make_float4(dc_low(acc[a][0]), dc_high(acc[a][0]), dc_low(acc[a][1]), dc_high(acc[a][1]));
#pragma unroll
          for (int z = 0; z < KG - 1; ++z) {
            const float4 p = *reinterpret_cast<const float4*>(part + z * DC_D * CS + idx);
            s = make_float4(s.x + p.x, s.y + p.y, s.z + p.z, s.w + p.w);
          }
          const float4 old = *reinterpret_cast<const float4*>(S + idx);
          *reinterpret_cast<float4*>(S + idx) = make_float4(fmaf(whole, old.x, s.x), fmaf(whole, old.y, s.y), fmaf(whole, old.z, s.z), fmaf(whole, old.w, s.w));
        }
      }
    }
  }
  __syncthreads();
  for (int idx = tid; idx < DC_D * CS; idx += DC_THREADS) {
    const int c = idx / CS, j = idx % CS;
    if (c < P.dk && j < cols) home[(size_t)c * P.dv + j] = S[idx];
  }
}

// total[i][..] += X[i][0 .. n) times Y[0 .. n)[the thread's columns 4 tx .. , 64 + 4 tx ..]; the sum over n is made by itself first.
// DIAGONAL: row i goes on to column n + i and leaves the rows of Y behind it out, whatever they hold (zero times an infinite value
// would not be zero).
template <bool DIAGONAL = false>
__device__ __forceinline__ void dc_rows_times(const float* X, int ldx, const float* Y, int n, int tx, u64 (&total)[4][4]) {
  u64 acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0ull;
#pragma unroll 2
  for (int c = 0; c < n; c += 4) {
    float4 x[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) x[i] = *reinterpret_cast<const float4*>(X + i * ldx + c);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const ulonglong2 y0 = *reinterpret_cast<const ulonglong2*>(Y + (c + e) * DC_D + 4 * tx), y1 = *reinterpret_cast<const ulonglong2*>(Y + (c + e) * DC_D + 64 + 4 * tx);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const u64 xx = dc_twice(e == 0 ? x[i].x : (e == 1 ? x[i].y : (e == 2 ? x[i].z : x[i].w)));
        acc[i][0] = dc_fma2(xx, y0.x, acc[i][0]);
        acc[i][1] = dc_fma2(xx, y0.y, acc[i][1]);
        acc[i][2] = dc_fma2(xx, y1.x, acc[i][2]);
        acc[i][3] = dc_fma2(xx, y1.y, acc[i][3]);
      }
    }
  }
  if (DIAGONAL)
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const ulonglong2 y0 = *reinterpret_cast<const ulonglong2*>(Y + (n + e) * DC_D + 4 * tx), y1 = *reinterpret_cast<const ulonglong2*>(Y + (n + e) * DC_D + 64 + 4 * tx);
#pragma unroll
      for (int i = e; i < 4; ++i) {
        const u64 xx = dc_twice(X[i * ldx + n + e]);
        acc[i][0] = dc_fma2(xx, y0.x, acc[i][0]);
        acc[i][1] = dc_fma2(xx, y0.y, acc[i][1]);
        acc[i][2] = dc_fma2(xx, y1.x, acc[i][2]);
        acc[i][3] = dc_fma2(xx, y1.y, acc[i][3]);
      }
    }
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) total[i][j] = dc_add2(total[i][j], acc[i][j]);
}

__global__ void __launch_bounds__(DC_THREADS, 2) delta_outputs_kernel(const __grid_constant__ DeltaChunkParams P) {
  JLX_TL(TL_OTHER);
  extern __shared__ __align__(16) float smem[];
  float* Q = smem;                  // [CHUNK][DC_LD]
  float* K = Q + CHUNK * DC_LD;     // [CHUNK][DC_LD]; then U: [CHUNK][DC_D]
  float* A = K + CHUNK * DC_LD;     // [10][PIECE][PIECE]: the pieces on and below the diagonal, (p, b) at p (p + 1) / 2 + b
  float* S = A + 10 * PIECE * PIECE;  // two quarters of the start state: [2][32][DC_D]
  __shared__ float g[CHUNK], from[CHUNK], to[CHUNK], piece[PIECES];
  const int chunk = blockIdx.x, h = blockIdx.y, tid = threadIdx.x;
  const int n0 = P.chunks[3 * chunk + 1], cnt = P.chunks[3 * chunk + 2] - n0;
  const int kh = h / (P.H / P.G);
  const size_t at = (size_t)chunk * P.H + h;
  dc_load(Q, DC_LD, P.q + ((size_t)n0 * P.G + kh) * P.dk, (size_t)P.G * P.dk, CHUNK, DC_D, cnt, P.dk);
  dc_load(K, DC_LD, P.k + ((size_t)n0 * P.G + kh) * P.dk, (size_t)P.G * P.dk, CHUNK, DC_D, cnt, P.dk);
  dc_commit();
  auto load_quarter = [&](int quarter) {  // 32 rows of the start state
    dc_load(S + (quarter & 1) * 32 * DC_D, DC_D, P.S0 + (at * P.dk + 32 * quarter) * P.dv, P.dv, 32, DC_D, max(0, P.dk - 32 * quarter), P.dv);
    dc_commit();
  };
  load_quarter(0);
  load_quarter(1);
  if (tid < CHUNK) g[tid] = tid < cnt ? P.decay[(size_t)(n0 + tid) * P.H + h] : 1.f;
  dc_wait<2>();
  __syncthreads();
  dc_products(g, from, to, piece);
  const int sl = tid & 15, tl = tid >> 4;
  float sum[PIECES][PIECES];
  dc_piece_products(Q, K, tl, sl, sum);
  __syncthreads();  // the keys are read, the products of decays are there
  dc_load(K, DC_D, P.X + at * CHUNK * P.dv, P.dv, CHUNK, DC_D, CHUNK, P.dv);
  dc_commit();
#pragma unroll
  for (int p = 0; p < PIECES; ++p)
#pragma unroll
    for (int b = 0; b <= p; ++b) {
      const int t = p * PIECE + tl, s = b * PIECE + sl;
      A[((p * (p + 1) / 2 + b) * PIECE + tl) * PIECE + sl] = s <= t ? dc_between(g, from, to, piece, t, s) * sum[p][b] : 0.f;
    }
  const int tx = tid & 15, ty = tid >> 4;
  u64 acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0ull;
  dc_wait<0>();
  __syncthreads();
#pragma unroll 1
  for (int quarter = 0; quarter < 4; ++quarter) {
    if (quarter >= 2) {
      if (quarter == 2) dc_wait<1>();
      else dc_wait<0>();
      __syncthreads();
    }
    if (4 * ty < cnt) dc_rows_times(Q + 4 * ty * DC_LD + 32 * quarter, DC_LD, S + (quarter & 1) * 32 * DC_D, 32, tx, acc);
    if (quarter < 2) {
      __syncthreads();
      load_quarter(quarter + 2);
    }
  }
  if (4 * ty >= cnt) return;
#pragma unroll
  for (int i = 0; i < 4; ++i) {  // the state's decay
    const u64 x = dc_twice(dc_from_start(from, piece, 4 * ty + i));
#pragma unroll
    for (int j = 0; j < 4; ++j) asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(acc[i][j]) : "l"(acc[i][j]), "l"(x));
  }
  const int p = ty / 4;
  for (int b = 0; b < p; ++b) dc_rows_times(A + ((p * (p + 1) / 2 + b) * PIECE + 4 * (ty & 3)) * PIECE, PIECE, K + b * PIECE * DC_D, PIECE, tx, acc);
  dc_rows_times<true>(A + (p * (p + 3) / 2 * PIECE + 4 * (ty & 3)) * PIECE, PIECE, K + p * PIECE * DC_D, 4 * (ty & 3), tx, acc);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int t = 4 * ty + i;
    if (t >= cnt) break;
    float* out = P.o + ((size_t)(n0 + t) * P.H + h) * P.dv;
#pragma unroll
    for (int hh = 0; hh < 2; ++hh) {
      const int j = 64 * hh + 4 * tx;
      if (j < P.dv)
        *reinterpret_cast<float4*>(out + j) = make_float4(dc_low(acc[i][2 * hh]), dc_high(acc[i][2 * hh]), dc_low(acc[i][2 * hh + 1]), dc_high(acc[i][2 * hh + 1]));
    }
  }
}

JLX_API int jlx_delta_chunk_supported(int dk, int dv) { return dk > 64 && dk <= DC_D && dv > 64 && dv <= DC_D && dk % 4 == 0 && dv % 4 == 0; }

// chunks: int32 [n, 3] (request, first token row, end row), at most 64 rows each; requests: int32 [m, 3] (request, first chunk,
// chunks), every chunk in exactly one.  All rows but the states' start on 16-byte boundaries.  scratch: n H (CHUNK (dk + dv + 1) +
// dk dv + 1) float32 elements.
JLX_API int jlx_delta_chunk(const float* q, const float* k, const float* v, const float* beta, const float* decay, float* state, const int* slot_ids,
                            float* o, const int* chunks, int n, const int* requests, int m, int G, int H, int dk, int dv, float* scratch,
                            cudaStream_t stream) {
  JLX_REQUIRE(n >= 0 && m >= 0 && G > 0 && H > 0 && H % G == 0, "delta_chunk: bad sizes n=%d m=%d G=%d H=%d", n, m, G, H);
  JLX_REQUIRE(jlx_delta_chunk_supported(dk, dv), "delta_chunk: heads of %d x %d are not supported", dk, dv);
  JLX_REQUIRE(H <= 65535, "delta_chunk: too many heads");
  if (n == 0 || m == 0) return 0;
  JLX_REQUIRE(scratch && (((uintptr_t)q | (uintptr_t)k | (uintptr_t)v | (uintptr_t)o | (uintptr_t)scratch) & 15) == 0,
              "delta_chunk: rows must start on 16-byte boundaries");
  float* X = scratch;
  float* Y = X + (size_t)n * H * CHUNK * dv;
  float* S0 = Y + (size_t)n * H * CHUNK * dk;
  float* ends = S0 + (size_t)n * H * dk * dv;
  float* wholes = ends + (size_t)n * H * CHUNK;
  const DeltaChunkParams P = {q, k, v, beta, decay, chunks, requests, slot_ids, state, o, X, Y, S0, ends, wholes, G, H, dk, dv};
  const int smem_solve = (int)sizeof(float) * (2 * CHUNK * DC_LD + CHUNK * DC_LDL);
  const int smem_out = (int)sizeof(float) * (2 * CHUNK * DC_LD + 10 * PIECE * PIECE + 2 * 32 * DC_D);
  const int smem_chain = (int)sizeof(float) * (2 * CHUNK * DC_LD + 3 * CHUNK * DC_CS + DC_D * DC_CS + 3 * DC_D * DC_CS);  // two blocks a multiprocessor
  JLX_CUDA(cudaFuncSetAttribute(delta_chain_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_chain));
  JLX_CUDA(cudaFuncSetAttribute(delta_solve_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_solve));
  JLX_CUDA(cudaFuncSetAttribute(delta_outputs_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_out));
  delta_solve_kernel<<<dim3(n, H), DC_THREADS, smem_solve, stream>>>(P);
  JLX_LAUNCH_CHECK("delta_solve");
  delta_chain_kernel<<<dim3(m, H, (dv + DC_CS - 1) / DC_CS), DC_THREADS, smem_chain, stream>>>(P);
  JLX_LAUNCH_CHECK("delta_chain");
  delta_outputs_kernel<<<dim3(n, H), DC_THREADS, smem_out, stream>>>(P);
  JLX_LAUNCH_CHECK("delta_outputs");
  return 0;
}
