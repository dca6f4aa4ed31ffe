// The decayed linear-attention recurrence of decay_scan.cu and recurrent.cu over long portions, by chunks of 64 tokens:
//
//     S_t = diag(d_t) S_(t-1) + k_t v_t^T,   o_t = S_t^T q_t   or   o_t = (S_(t-1) + diag(u) k_t v_t^T)^T q_t.
//
// Walked token by token, a request's prompt is a chain of as many dependent steps on the few blocks that its state fills.
// With chunks (the chunkwise form of S. Yang et al., "Gated Linear Attention Transformers with Hardware-Efficient Training", 2023)
// almost all of it is products of 64 rows, over all chunks and heads at once:
//
//   chunk_states   what a chunk adds to a zero state, sum_t (k_t prod_{r>t} d_r) v_t^T, and the product of its decays.
//   chunk_chain    the chunks' start states, S <- diag(prod d) S + added, chunk after chunk (the one dependent chain, of
//                  elementwise steps); the last one becomes the request's state.
//   chunk_outputs  o_t = (q_t prod_{r<=t} d_r)^T S_start + sum_{s<=t} A_ts v_s,
//                  A_ts = sum_c q_tc k_sc prod_{s<r<=t} d_rc (read before the update: r < t, and u in the place of the
//                  product for s = t).
//
// Decays may be as small as they like: no quotient of products is taken.  A is made in pieces of 16 x 16: on the diagonal
// each k_s is decayed step by step; below it the rows of q are decayed from their piece's start and the rows of k to their
// piece's end and on, piece by piece, to the start of q's.  Everything is 32-bit (two FMAs per instruction).  A token's sums
// depend on where it stands in its chunk, and chunks count from the request's first token of the step: cutting a prompt
// elsewhere moves the last bits of a result, no more.
// Bound by 32-bit FMAs (2 x 128 x 128 per token and head for the two products, and about half as many for A) and, in
// chunk_outputs, by the shared-memory reads and shuffles of A's diagonal.  One request of 2048 tokens, 16 heads of 128 x 128:
// states 36 us, chain 16, outputs 84, together 144 (the token-by-token walk: 297); 32 heads: 263 (398).
#include "common.cuh"

#define CHUNK 64
#define PIECE 16
#define CH_D 128     // channels and value columns a head may have (zeros beyond its own)
#define CH_LD 132    // row of q, k, d in shared memory: eight rows start in eight different 16-byte columns of banks
#define CH_THREADS 256

struct ChunkRows {  // element (token, head, i) = p[token * ld + head * size + i]
  const float* p;
  long long ld;
};

struct ChunkParams {
  ChunkRows q, k, d, v;  // k.p null: k = 1 - d
  const float* bonus;    // [H, dk]; used when read before the update (null: none)
  const int* chunks;     // [n, 3]: request, first token row, end row; a request's chunks in order
  const int* requests;   // [m, 3]: request, its first chunk, its chunks
  const int* slot_ids;
  float* state;          // [slots, H, dk, dv]
  float* o;              // [N, H, dv]
  float* added;          // [n, H, dk, dv]: what a chunk adds; then its start state
  float* decay;          // [n, H, dk]: the product of its decays
  int H, dk, dv, vec;    // vec: every row piece starts on 16 bytes and sizes are multiples of 4
};

__device__ __forceinline__ unsigned long long ch_fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
  unsigned long long r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
typedef unsigned long long u64;
__device__ __forceinline__ u64 ch_mul2(u64 a, u64 b) {
  u64 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ u64 ch_pair(float x, float y) { return (u64)__float_as_uint(x) | ((u64)__float_as_uint(y) << 32); }
__device__ __forceinline__ unsigned long long ch_twice(float x) {
  return (unsigned long long)__float_as_uint(x) | ((unsigned long long)__float_as_uint(x) << 32);
}
__device__ __forceinline__ float ch_low(unsigned long long p) { return __uint_as_float((unsigned)p); }
__device__ __forceinline__ float ch_high(unsigned long long p) { return __uint_as_float((unsigned)(p >> 32)); }
__device__ __forceinline__ void ch_copy16(float* dst, const float* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void ch_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void ch_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// A chunk's rows of one operand into shared memory [CHUNK][ld], `fill` where the chunk or the head ends.
__device__ __forceinline__ void ch_load(float* dst, int ld, const ChunkRows& rows, int n0, int cnt, int head, int size, float fill, int vec) {
  for (int idx = threadIdx.x; idx < CHUNK * (CH_D / 4); idx += CH_THREADS) {
    const int t = idx / (CH_D / 4), c = idx % (CH_D / 4) * 4;
    float* to = dst + t * ld + c;
    const float* from = rows.p + (size_t)(n0 + t) * rows.ld + (size_t)head * size + c;
    if (vec && t < cnt && c < size) {
      ch_copy16(to, from);
    } else {
#pragma unroll
      for (int e = 0; e < 4; ++e) to[e] = t < cnt && c + e < size ? from[e] : fill;
    }
  }
}
// k = 1 - d, for the chunk's own rows and channels (zeros elsewhere: d is one there)
__device__ __forceinline__ void ch_one_minus(float* k, const float* d) {
  for (int idx = threadIdx.x; idx < CHUNK * CH_D; idx += CH_THREADS) {
    const int at = idx / CH_D * CH_LD + idx % CH_D;
    k[at] = 1.f - d[at];
  }
}

__global__ void __launch_bounds__(CH_THREADS, 2) chunk_states_kernel(const __grid_constant__ ChunkParams P) {
  JLX_TL(TL_OTHER);
  extern __shared__ __align__(16) float smem[];
  float* K = smem;                  // [CHUNK][CH_LD]
  float* D = K + CHUNK * CH_LD;     // [CHUNK][CH_LD]
  float* V = D + CHUNK * CH_LD;     // [CHUNK][CH_D]
  const int chunk = blockIdx.x, head = blockIdx.y, tid = threadIdx.x;
  const int n0 = P.chunks[3 * chunk + 1], cnt = P.chunks[3 * chunk + 2] - n0;
  if (P.k.p) ch_load(K, CH_LD, P.k, n0, cnt, head, P.dk, 0.f, P.vec);
  ch_load(D, CH_LD, P.d, n0, cnt, head, P.dk, 1.f, P.vec);
  ch_commit();
  ch_load(V, CH_D, P.v, n0, cnt, head, P.dv, 0.f, P.vec);
  ch_commit();
  ch_wait<1>();
  __syncthreads();
  if (!P.k.p) {
    ch_one_minus(K, D);
    __syncthreads();
  }
  // two halves of the chunk at once: each k decayed to its half's end, then the first half's to the chunk's
  __shared__ float half_decay[CH_D];
  {
    const int c = tid & (CH_D - 1), h = tid >> 7;
    float suffix = 1.f;
#pragma unroll 8
    for (int t = CHUNK / 2 * (h + 1) - 1; t >= CHUNK / 2 * h; --t) {
      K[t * CH_LD + c] *= suffix;
      suffix *= D[t * CH_LD + c];
    }
    if (h == 1) half_decay[c] = suffix;
    __syncthreads();
    if (h == 0) {
      const float later = half_decay[c];
#pragma unroll 8
      for (int t = 0; t < CHUNK / 4; ++t) K[t * CH_LD + c] *= later;
      if (c < P.dk) P.decay[((size_t)chunk * P.H + head) * P.dk + c] = suffix * later;
    } else {
      const float later = half_decay[c];
#pragma unroll 8
      for (int t = CHUNK / 4; t < CHUNK / 2; ++t) K[t * CH_LD + c] *= later;
    }
  }
  ch_wait<0>();
  __syncthreads();
  // [channels][value columns] += k v^T: eight channels (4 ty, 64 + 4 ty) by eight columns (4 tx, 64 + 4 tx) per thread
  const int tx = tid & 15, ty = tid >> 4;
  unsigned long long acc[8][4];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0ull;
#pragma unroll 2
  for (int t = 0; t < CHUNK; ++t) {
    const float4 k0 = *reinterpret_cast<const float4*>(K + t * CH_LD + 4 * ty), k1 = *reinterpret_cast<const float4*>(K + t * CH_LD + 64 + 4 * ty);
    const ulonglong2 v0 = *reinterpret_cast<const ulonglong2*>(V + t * CH_D + 4 * tx), v1 = *reinterpret_cast<const ulonglong2*>(V + t * CH_D + 64 + 4 * tx);
    const float k[8] = {k0.x, k0.y, k0.z, k0.w, k1.x, k1.y, k1.z, k1.w};
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const unsigned long long x = ch_twice(k[i]);
      acc[i][0] = ch_fma2(x, v0.x, acc[i][0]);
      acc[i][1] = ch_fma2(x, v0.y, acc[i][1]);
      acc[i][2] = ch_fma2(x, v1.x, acc[i][2]);
      acc[i][3] = ch_fma2(x, v1.y, acc[i][3]);
    }
  }
  float* out = P.added + ((size_t)chunk * P.H + head) * P.dk * P.dv;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int c = (i < 4 ? 0 : 64) + 4 * ty + (i & 3);
    if (c >= P.dk) continue;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int j = 64 * h + 4 * tx;
      const float v[4] = {ch_low(acc[i][2 * h]), ch_high(acc[i][2 * h]), ch_low(acc[i][2 * h + 1]), ch_high(acc[i][2 * h + 1])};
      if ((P.dv & 3) == 0) {
        if (j < P.dv) *reinterpret_cast<float4*>(out + (size_t)c * P.dv + j) = make_float4(v[0], v[1], v[2], v[3]);
      } else {
#pragma unroll
        for (int e = 0; e < 4; ++e)
          if (j + e < P.dv) out[(size_t)c * P.dv + j + e] = v[e];
      }
    }
  }
}

// One thread per state entry of a request, eight chunks' entries in flight at once.
__global__ void __launch_bounds__(256) chunk_chain_kernel(const __grid_constant__ ChunkParams P) {
  JLX_TL(TL_OTHER);
  const int r = P.requests[3 * blockIdx.y], first = P.requests[3 * blockIdx.y + 1], count = P.requests[3 * blockIdx.y + 2];
  const size_t size = (size_t)P.H * P.dk * P.dv, i = (size_t)blockIdx.x * 256 + threadIdx.x;
  if (i >= size) return;
  const size_t row = i / P.dv, rows = (size_t)P.H * P.dk;
  float* home = P.state + (size_t)P.slot_ids[r] * size + i;
  float* a = P.added + (size_t)first * size + i;
  const float* d = P.decay + (size_t)first * rows + row;
  float s = *home;
  constexpr int AHEAD = 8;
  for (int c0 = 0; c0 < count; c0 += AHEAD) {
    float x[AHEAD], y[AHEAD];
#pragma unroll
    for (int u = 0; u < AHEAD; ++u) {
      const bool there = c0 + u < count;
      x[u] = there ? a[(size_t)(c0 + u) * size] : 0.f;
      y[u] = there ? d[(size_t)(c0 + u) * rows] : 1.f;
    }
#pragma unroll
    for (int u = 0; u < AHEAD; ++u)
      if (c0 + u < count) {
        a[(size_t)(c0 + u) * size] = s;
        s = fmaf(y[u], s, x[u]);
      }
  }
  *home = s;
}

// acc[i][..] += X[i][0 .. n) times Y[0 .. n)[the thread's columns 4 tx .. , 64 + 4 tx ..]
__device__ __forceinline__ void ch_rows_times(const float* X, int ldx, const float* Y, int n, int tx, unsigned long long (&acc)[4][4]) {
#pragma unroll 2
  for (int c = 0; c < n; c += 4) {
    float4 x[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) x[i] = *reinterpret_cast<const float4*>(X + i * ldx + c);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const ulonglong2 y0 = *reinterpret_cast<const ulonglong2*>(Y + (c + e) * CH_D + 4 * tx), y1 = *reinterpret_cast<const ulonglong2*>(Y + (c + e) * CH_D + 64 + 4 * tx);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const unsigned long long xx = ch_twice(e == 0 ? x[i].x : (e == 1 ? x[i].y : (e == 2 ? x[i].z : x[i].w)));
        acc[i][0] = ch_fma2(xx, y0.x, acc[i][0]);
        acc[i][1] = ch_fma2(xx, y0.y, acc[i][1]);
        acc[i][2] = ch_fma2(xx, y1.x, acc[i][2]);
        acc[i][3] = ch_fma2(xx, y1.y, acc[i][3]);
      }
    }
  }
}

// The same for four rows of a diagonal piece, whose first is column n: row n + i takes the columns up to its own and leaves the rows
// of Y behind them out, whatever they hold (zero times an infinite value would not be zero).
__device__ __forceinline__ void ch_rows_times_to_diagonal(const float* X, const float* Y, int n, int tx, unsigned long long (&acc)[4][4]) {
  ch_rows_times(X, PIECE, Y, n, tx, acc);
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const ulonglong2 y0 = *reinterpret_cast<const ulonglong2*>(Y + (n + e) * CH_D + 4 * tx), y1 = *reinterpret_cast<const ulonglong2*>(Y + (n + e) * CH_D + 64 + 4 * tx);
#pragma unroll
    for (int i = e; i < 4; ++i) {
      const unsigned long long xx = ch_twice(X[i * PIECE + n + e]);
      acc[i][0] = ch_fma2(xx, y0.x, acc[i][0]);
      acc[i][1] = ch_fma2(xx, y0.y, acc[i][1]);
      acc[i][2] = ch_fma2(xx, y1.x, acc[i][2]);
      acc[i][3] = ch_fma2(xx, y1.y, acc[i][3]);
    }
  }
}

template <bool READ_AFTER>
__global__ void __launch_bounds__(CH_THREADS, 2) chunk_outputs_kernel(const __grid_constant__ ChunkParams P) {
  JLX_TL(TL_OTHER);
  extern __shared__ __align__(16) float smem[];
  float* Q = smem;                  // [CHUNK][CH_LD]
  float* K = Q + CHUNK * CH_LD;     // [CHUNK][CH_LD]; then quarters of the start state, two at a time: [2][32][CH_D]
  float* D = K + CHUNK * CH_LD;     // [CHUNK][CH_LD]; then v: [CHUNK][CH_D]
  float* A = D + CHUNK * CH_LD;     // [10][PIECE][PIECE]: the pieces on and below the diagonal, (p, b) at p (p + 1) / 2 + b
  float* tot = A + 10 * PIECE * PIECE;  // [CHUNK / PIECE - 1][CH_D]: the products of the pieces' decays
  float* V = D;
  const int chunk = blockIdx.x, head = blockIdx.y, tid = threadIdx.x;
  const int n0 = P.chunks[3 * chunk + 1], cnt = P.chunks[3 * chunk + 2] - n0;
  ch_load(Q, CH_LD, P.q, n0, cnt, head, P.dk, 0.f, P.vec);
  if (P.k.p) ch_load(K, CH_LD, P.k, n0, cnt, head, P.dk, 0.f, P.vec);
  ch_load(D, CH_LD, P.d, n0, cnt, head, P.dk, 1.f, P.vec);
  ch_commit();
  const float* start = P.added + ((size_t)chunk * P.H + head) * P.dk * P.dv;
  auto load_quarter = [&](int quarter) {  // 32 rows of the start state
    float* to = K + (quarter & 1) * 32 * CH_D;
    for (int idx = tid; idx < 32 * (CH_D / 4); idx += CH_THREADS) {
      const int cl = idx / (CH_D / 4), c = 32 * quarter + cl, j = idx % (CH_D / 4) * 4;
      if ((P.dv & 3) == 0 && c < P.dk && j < P.dv) {
        ch_copy16(to + cl * CH_D + j, start + (size_t)c * P.dv + j);
      } else {
#pragma unroll
        for (int e = 0; e < 4; ++e) to[cl * CH_D + j + e] = c < P.dk && j + e < P.dv ? start[(size_t)c * P.dv + j + e] : 0.f;
      }
    }
    ch_commit();
  };
  ch_wait<0>();
  __syncthreads();
  if (!P.k.p) {
    ch_one_minus(K, D);
    __syncthreads();
  }
  // A on the diagonal: a thread decays k_s and k_(s + 8), eight channels (4 g .., 64 + 4 g ..) of each, from token to token;
  // half of the block takes the even pieces, half the odd ones
  {
    const int g = tid & 15, sl = (tid >> 4) & 7;
    u64 u[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int c = (e < 2 ? 0 : 64) + 4 * g + 2 * (e & 1);
      auto bonus = [&](int i) { return !READ_AFTER && P.bonus && i < P.dk ? P.bonus[head * P.dk + i] : 0.f; };
      u[e] = ch_pair(bonus(c), bonus(c + 1));
    }
    auto eight = [&](const float* row, u64 (&x)[4]) {
      const ulonglong2 lo = *reinterpret_cast<const ulonglong2*>(row + 4 * g), hi = *reinterpret_cast<const ulonglong2*>(row + 64 + 4 * g);
      x[0] = lo.x; x[1] = lo.y; x[2] = hi.x; x[3] = hi.y;
    };
#pragma unroll 1
    for (int p = tid >> 7; p < CHUNK / PIECE; p += 2) {
      float* out = A + p * (p + 3) / 2 * PIECE * PIECE;
      u64 w[2][4];
#pragma unroll
      for (int x = 0; x < 2; ++x) eight(K + (p * PIECE + sl + 8 * x) * CH_LD, w[x]);
#pragma unroll 2
      for (int t0 = 0; t0 < PIECE; t0 += 2) {
        float v[2][2];  // [token][s]
#pragma unroll
        for (int tt = 0; tt < 2; ++tt) {
          const int tl = t0 + tt;
          u64 q[4], d[4];
          eight(Q + (p * PIECE + tl) * CH_LD, q);
          eight(D + (p * PIECE + tl) * CH_LD, d);
#pragma unroll
          for (int x = 0; x < 2; ++x) {
            const int s = sl + 8 * x;
            u64 sum = 0ull;
            if (READ_AFTER && tl > s)
#pragma unroll
              for (int e = 0; e < 4; ++e) w[x][e] = ch_mul2(w[x][e], d[e]);
            if (!READ_AFTER && tl == s) {
#pragma unroll
              for (int e = 0; e < 4; ++e) sum = ch_fma2(q[e], ch_mul2(u[e], w[x][e]), sum);
            } else {
#pragma unroll
              for (int e = 0; e < 4; ++e) sum = ch_fma2(q[e], w[x][e], sum);
            }
            if (!READ_AFTER && tl > s)
#pragma unroll
              for (int e = 0; e < 4; ++e) w[x][e] = ch_mul2(w[x][e], d[e]);
            v[tt][x] = ch_low(sum) + ch_high(sum);
          }
        }
        // sixteen lanes add four numbers in five exchanges: each step halves the numbers a lane still carries
        const bool up8 = g & 8, up4 = g & 4;
        float y[2];
#pragma unroll
        for (int x = 0; x < 2; ++x) y[x] = (up8 ? v[1][x] : v[0][x]) + __shfl_xor_sync(0xffffffffu, up8 ? v[0][x] : v[1][x], 8);
        float z = (up4 ? y[1] : y[0]) + __shfl_xor_sync(0xffffffffu, up4 ? y[0] : y[1], 4);
        z += __shfl_xor_sync(0xffffffffu, z, 2);
        z += __shfl_xor_sync(0xffffffffu, z, 1);
        const int t = t0 + (up8 ? 1 : 0), s = sl + (up4 ? 8 : 0);
        if ((g & 3) == 0) out[t * PIECE + s] = t >= s ? z : 0.f;
      }
    }
  }
  __syncthreads();
  // rows of q decayed from their piece's start, rows of k to their piece's end; the pieces' own products
  {
    const int c = tid & (CH_D - 1), half = tid >> 7;
    if (half == 0) {
#pragma unroll 1
      for (int p = 0; p < CHUNK / PIECE; ++p) {
        float prefix = 1.f;
#pragma unroll
        for (int t = p * PIECE; t < (p + 1) * PIECE; ++t) {
          const float d = D[t * CH_LD + c];
          if (READ_AFTER) prefix *= d;
          Q[t * CH_LD + c] *= prefix;
          if (!READ_AFTER) prefix *= d;
        }
        if (p < CHUNK / PIECE - 1) tot[p * CH_D + c] = prefix;
      }
    } else {
#pragma unroll 1
      for (int p = 0; p < CHUNK / PIECE - 1; ++p) {  // (no row of q lies behind the last piece)
        float suffix = 1.f;
#pragma unroll
        for (int t = (p + 1) * PIECE - 1; t >= p * PIECE; --t) {
          K[t * CH_LD + c] *= suffix;
          suffix *= D[t * CH_LD + c];
        }
      }
    }
  }
  __syncthreads();
  ch_load(V, CH_D, P.v, n0, cnt, head, P.dv, 0.f, P.vec);  // the decays are read: their place serves the values
  ch_commit();
  // A below the diagonal: piece row p against the pieces before it, thread (t, s mod 16)
#pragma unroll 1
  for (int p = 1; p < CHUNK / PIECE; ++p) {
    const int sl = tid & 15, tl = tid >> 4;
    if (p > 1) {  // the pieces before the last one are decayed over it
      const int c = 4 * (tid & 31);
      const ulonglong2 by = *reinterpret_cast<const ulonglong2*>(tot + (p - 1) * CH_D + c);
      for (int t = tid >> 5; t < (p - 1) * PIECE; t += CH_THREADS / 32) {
        ulonglong2* k = reinterpret_cast<ulonglong2*>(K + t * CH_LD + c);
        *k = make_ulonglong2(ch_mul2(k->x, by.x), ch_mul2(k->y, by.y));
      }
      __syncthreads();
    }
    unsigned long long sum[3] = {0ull, 0ull, 0ull};
    const float* q = Q + (p * PIECE + tl) * CH_LD;
#pragma unroll 4
    for (int c = 0; c < CH_D; c += 4) {
      const ulonglong2 x = *reinterpret_cast<const ulonglong2*>(q + c);
#pragma unroll
      for (int b = 0; b < 3; ++b)
        if (b < p) {
          const ulonglong2 y = *reinterpret_cast<const ulonglong2*>(K + (b * PIECE + sl) * CH_LD + c);
          sum[b] = ch_fma2(x.y, y.y, ch_fma2(x.x, y.x, sum[b]));
        }
    }
#pragma unroll
    for (int b = 0; b < 3; ++b)
      if (b < p) A[((p * (p + 1) / 2 + b) * PIECE + tl) * PIECE + sl] = ch_low(sum[b]) + ch_high(sum[b]);
    __syncthreads();
  }
  load_quarter(0);  // the keys are read: their place serves the start state
  load_quarter(1);
  // rows of q decayed from the chunk's start
  {
    const int c = 4 * (tid & 31);
    ulonglong2 before = *reinterpret_cast<const ulonglong2*>(tot + c);
#pragma unroll
    for (int p = 1; p < CHUNK / PIECE; ++p) {
      for (int t = p * PIECE + (tid >> 5); t < (p + 1) * PIECE; t += CH_THREADS / 32) {
        ulonglong2* q = reinterpret_cast<ulonglong2*>(Q + t * CH_LD + c);
        *q = make_ulonglong2(ch_mul2(q->x, before.x), ch_mul2(q->y, before.y));
      }
      if (p + 1 < CHUNK / PIECE) {
        const ulonglong2 by = *reinterpret_cast<const ulonglong2*>(tot + p * CH_D + c);
        before = make_ulonglong2(ch_mul2(before.x, by.x), ch_mul2(before.y, by.y));
      }
    }
  }
  const int tx = tid & 15, ty = tid >> 4;
  unsigned long long acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0ull;
#pragma unroll 1
  for (int quarter = 0; quarter < 4; ++quarter) {
    if (quarter < 3) ch_wait<1>();
    else ch_wait<0>();
    __syncthreads();  // this quarter is there (and the values, and with the first one all of q)
    if (4 * ty < cnt) ch_rows_times(Q + 4 * ty * CH_LD + 32 * quarter, CH_LD, K + (quarter & 1) * 32 * CH_D, 32, tx, acc);
    if (quarter < 2) {
      __syncthreads();
      load_quarter(quarter + 2);
    }
  }
  if (4 * ty >= cnt) return;
  const int p = ty / 4;
  for (int b = 0; b < p; ++b)
    ch_rows_times(A + ((p * (p + 1) / 2 + b) * PIECE + 4 * (ty & 3)) * PIECE, PIECE, V + b * PIECE * CH_D, PIECE, tx, acc);
  ch_rows_times_to_diagonal(A + (p * (p + 3) / 2 * PIECE + 4 * (ty & 3)) * PIECE, V + p * PIECE * CH_D, 4 * (ty & 3), tx, acc);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int t = 4 * ty + i;
    if (t >= cnt) break;
    float* out = P.o + ((size_t)(n0 + t) * P.H + head) * P.dv;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int j = 64 * h + 4 * tx;
      const float v[4] = {ch_low(acc[i][2 * h]), ch_high(acc[i][2 * h]), ch_low(acc[i][2 * h + 1]), ch_high(acc[i][2 * h + 1])};
      if ((P.dv & 3) == 0) {
        if (j < P.dv) *reinterpret_cast<float4*>(out + j) = make_float4(v[0], v[1], v[2], v[3]);
      } else {
#pragma unroll
        for (int e = 0; e < 4; ++e)
          if (j + e < P.dv) out[j + e] = v[e];
      }
    }
  }
}

// chunks: int32 [n, 3] (request, first token row, end row), at most 64 rows each; requests: int32 [m, 3] (request, first chunk,
// chunks), every chunk in exactly one.  q, k, d, v: row pointers and strides (k null: k = 1 - d); o: [N, H, dv].  scratch: n H dk
// (dv + 1) float32 elements.
JLX_API int jlx_chunk_scan(const float* q, long long ldq, const float* k, long long ldk, const float* d, long long ldd, const float* v,
                           long long ldv, const float* bonus, float* state, const int* slot_ids, float* o, const int* chunks, int n,
                           const int* requests, int m, int H, int dk, int dv, int read_after, float* scratch, cudaStream_t stream) {
  JLX_REQUIRE(n >= 0 && m >= 0 && H > 0 && dk > 0 && dv > 0, "chunk_scan: bad sizes n=%d m=%d H=%d dk=%d dv=%d", n, m, H, dk, dv);
  JLX_REQUIRE(dk <= CH_D && dv <= CH_D, "chunk_scan: heads of %d x %d; up to %d x %d are supported", dk, dv, CH_D, CH_D);
  JLX_REQUIRE(H <= 65535 && m <= 65535, "chunk_scan: too many heads or requests");
  if (n == 0 || m == 0) return 0;
  JLX_REQUIRE(scratch && ((uintptr_t)scratch & 15) == 0 && ((uintptr_t)o & 15) == 0, "chunk_scan: scratch and output must start on 16 bytes");
  const uintptr_t at = (uintptr_t)q | (uintptr_t)k | (uintptr_t)d | (uintptr_t)v;
  const int vec = ((ldq | ldk | ldd | ldv | dk | dv) & 3) == 0 && (at & 15) == 0;
  const ChunkParams P = {{q, ldq}, {k, ldk}, {d, ldd}, {v, ldv}, bonus, chunks, requests, slot_ids, state, o, scratch, scratch + (size_t)n * H * dk * dv,
                         H, dk, dv, vec};
  const int smem_states = (int)sizeof(float) * (2 * CHUNK * CH_LD + CHUNK * CH_D);
  const int smem_out = (int)sizeof(float) * (3 * CHUNK * CH_LD + 10 * PIECE * PIECE + (CHUNK / PIECE - 1) * CH_D);  // two blocks an SM
  JLX_CUDA(cudaFuncSetAttribute(chunk_states_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_states));
  const auto outputs = read_after ? chunk_outputs_kernel<true> : chunk_outputs_kernel<false>;
  JLX_CUDA(cudaFuncSetAttribute(outputs, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_out));
  chunk_states_kernel<<<dim3(n, H), CH_THREADS, smem_states, stream>>>(P);
  JLX_LAUNCH_CHECK("chunk_states");
  chunk_chain_kernel<<<dim3((unsigned)(((size_t)H * dk * dv + 255) / 256), m), 256, 0, stream>>>(P);
  JLX_LAUNCH_CHECK("chunk_chain");
  outputs<<<dim3(n, H), CH_THREADS, smem_out, stream>>>(P);
  JLX_LAUNCH_CHECK("chunk_outputs");
  return 0;
}
