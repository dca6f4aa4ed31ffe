// Paged attention for any head size, head count, group size, page size and query length, in 32-bit
// or bfloat16 storage with 32-bit scores, softmax and accumulation.  It is the attention of the
// 32-bit path and the fallback of the bfloat16 path for sizes that the tensor-core kernels refuse.
//
// One block serves one query token and one KV head (all G query heads of the group share each key
// and value tile).  A query at position p of request r attends keys at positions [start, p] with
//   start = max(chunk  ? floor(p / chunk) * chunk : 0,  window ? p - window + 1 : 0)
// (causal and same-chunk mask of llama4/llama4_jax/model.py:731-742; scale dh^-0.5, model.py:774;
// 32-bit softmax, model.py:789).  Queries of layers with temperature tuning are scaled by
// 1 + attn_scale * ln(1 + floor((p + 1) / floor_scale)).
// With `keep` > 0 (and a window) the first `keep` keys of the sequence are visible besides the window's.
// With `sink` (one number per query head) the softmax has one more term in its denominator, exp(sink[h]), which
// carries no value: weights p_j = exp(s_j) / (exp(sink) + sum_i exp(s_i)); a sink of 0 adds one to the denominator.
// With `slopes` (one number per query head) slopes[h] * (p - j) is taken off the scaled score of key j: a bias that
// grows with the distance.
// With `softcap` > 0 the scaled score s becomes softcap * tanh(s / softcap) (before the bias and the sink).
// The order of the key loop depends only on (start, p): a position's result does not change with
// what else is in the batch or how the prompt was cut into steps.
#include "attention_maps.cuh"
#include "common.cuh"

#include <type_traits>

#define ATT_TILE 32
#define ATT_MAX_WARPS 8
#define ATT_MAX_D32 16  // head size up to 512

template <typename T, typename TO>
__global__ void attention_generic_kernel(const T* __restrict__ q, const T* __restrict__ pages,
                                         const int* __restrict__ block_table, int bt_stride,
                                         const int* __restrict__ req_of_token, const int* __restrict__ positions,
                                         TO* __restrict__ out, int Hq, int Hkv, int dh, int page_size, int num_pages,
                                         float scale, int chunk, int window, int keep, float attn_scale, float floor_scale,
                                         const float* __restrict__ sink, const float* __restrict__ slopes, float softcap,
                                         int* status) {
  JLX_TL(TL_ATTN_GENERIC);
  extern __shared__ float smem[];
  const int n = blockIdx.x, hk = blockIdx.y;
  const int G = Hq / Hkv;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
  const int ldk = dh + 1;
  float* qs = smem;                        // [nwarp][dh]
  float* ks = qs + nwarp * dh;             // [ATT_TILE][dh + 1]
  float* vs = ks + ATT_TILE * ldk;         // [ATT_TILE][dh + 1]

  const int p = positions[n];
  const int r = req_of_token[n];
  int start = 0;
  if (chunk > 0) start = (p / chunk) * chunk;
  if (window > 0) start = max(start, p - window + 1);
  const int kept = min(keep, start);  // kept keys below the window
  float qscale = scale;
  if (attn_scale != 0.f) qscale *= 1.f + attn_scale * log1pf(floorf(((float)p + 1.f) / floor_scale));
  const int nd = (dh + 31) >> 5;
  const size_t page_elems = (size_t)2 * Hkv * page_size * dh;

  for (int g0 = 0; g0 < G; g0 += nwarp) {
    const int g = g0 + warp;
    const bool active = g < G;
    const int h = hk * G + g;
    if (active)
      for (int d = lane; d < dh; d += 32) qs[warp * dh + d] = to_f32<T>(q[((size_t)n * Hq + h) * dh + d]);
    const float slope = slopes && active ? slopes[h] : 0.f;
    float m = -INFINITY, l = 0.f;
    float acc[ATT_MAX_D32];
#pragma unroll
    for (int i = 0; i < ATT_MAX_D32; ++i) acc[i] = 0.f;

    int t0 = kept > 0 ? 0 : start;
    while (t0 <= p) {
      __syncthreads();  // previous tile fully consumed; qs visible
      const int cnt = min(ATT_TILE, t0 < start ? kept - t0 : p - t0 + 1);
      for (int idx = threadIdx.x; idx < cnt * dh; idx += blockDim.x) {
        const int j = idx / dh, d = idx - j * dh;
        const int pos = t0 + j;
        const int page = block_table[(size_t)r * bt_stride + pos / page_size];
        float kv = 0.f, vv = 0.f;
        if (page < 0 || page >= num_pages) {
          atomicOr(status, JLX_STATUS_BAD_PAGE);
        } else {
          const T* base = pages + (size_t)page * page_elems + ((size_t)hk * page_size + pos % page_size) * dh + d;
          kv = to_f32<T>(base[0]);
          vv = to_f32<T>(base[(size_t)Hkv * page_size * dh]);
        }
        ks[j * ldk + d] = kv;
        vs[j * ldk + d] = vv;
      }
      __syncthreads();
      if (active) {
        float s = -INFINITY;
        if (lane < cnt) {
          float dot = 0.f;
          const float* kr = ks + lane * ldk;
          const float* qr = qs + warp * dh;
          for (int d = 0; d < dh; ++d) dot += qr[d] * kr[d];
          s = dot * qscale;
          if (softcap > 0.f) s = softcap * tanhf(s / softcap);
          s = fmaf(-slope, (float)(p - (t0 + lane)), s);
        }
        const float m_new = fmaxf(m, warp_max(s));
        const float corr = expf(m - m_new);  // m = -inf on the first tile: exp(-inf) = 0
        const float pj = lane < cnt ? expf(s - m_new) : 0.f;
        l = l * corr + warp_sum(pj);
        m = m_new;
#pragma unroll
        for (int i = 0; i < ATT_MAX_D32; ++i) {
          if (i < nd) {
            const int d = lane + 32 * i;
            float a = acc[i] * corr;
            for (int j = 0; j < cnt; ++j) {
              const float pv = __shfl_sync(0xffffffffu, pj, j);
              if (d < dh) a += pv * vs[j * ldk + d];
            }
            acc[i] = a;
          }
        }
      }
      t0 += ATT_TILE;
      if (t0 - ATT_TILE < start && t0 >= kept) t0 = start;  // the kept keys are through: on to the window
    }
    if (active) {
      float corr = 1.f;
      if (sink) {  // the sink joins the sum like a last key without a value
        const float m_new = fmaxf(m, sink[h]);
        corr = expf(m - m_new);
        l = l * corr + expf(sink[h] - m_new);
      }
#pragma unroll
      for (int i = 0; i < ATT_MAX_D32; ++i) {
        const int d = lane + 32 * i;
        if (i < nd && d < dh) out[((size_t)n * Hq + h) * dh + d] = from_f32<TO>(acc[i] * corr / l);
      }
    }
    __syncthreads();
  }
}

JLX_API int jlx_attention_generic(const void* q, const void* pages, int dtype, const int* block_table, int bt_stride,
                                  const int* req_of_token, const int* positions, void* out, int out_dtype, int N, int Hq, int Hkv,
                                  int dh, int page_size, int num_pages, float scale, int chunk, int window, int keep,
                                  float attn_scale, float floor_scale, const float* sink, const float* slopes,
                                  float softcap, int* status, cudaStream_t stream) {
  JLX_REQUIRE(N >= 0 && Hq > 0 && Hkv > 0 && dh > 0 && page_size > 0 && num_pages > 0, "attention: bad sizes");
  JLX_REQUIRE(Hq % Hkv == 0, "attention: %d query heads are no multiple of %d KV heads", Hq, Hkv);
  JLX_REQUIRE(dh <= 32 * ATT_MAX_D32, "attention: head size %d is above the supported maximum %d", dh, 32 * ATT_MAX_D32);
  JLX_REQUIRE(softcap >= 0.f, "attention: the score cap must be positive (0: none)");
  JLX_REQUIRE(attn_scale == 0.f || floor_scale > 0.f, "attention: floor_scale must be positive");
  if (N == 0) return 0;
  const int G = Hq / Hkv;
  const int nwarp = G < ATT_MAX_WARPS ? G : ATT_MAX_WARPS;
  const size_t smem = sizeof(float) * ((size_t)nwarp * dh + 2 * (size_t)ATT_TILE * (dh + 1));
  JLX_REQUIRE(Hkv <= 65535, "attention: too many KV heads (%d)", Hkv);
  JLX_REQUIRE(keep >= 0, "attention: the count of kept first keys is negative");
  JLX_DISPATCH_DTYPE(dtype, T, JLX_DISPATCH_DTYPE(out_dtype, TO, {
    if (smem > 48 * 1024)
      JLX_CUDA(cudaFuncSetAttribute(attention_generic_kernel<T, TO>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    attention_generic_kernel<T, TO><<<dim3(N, Hkv), nwarp * 32, smem, stream>>>(
        (const T*)q, (const T*)pages, block_table, bt_stride, req_of_token, positions, (TO*)out, Hq, Hkv, dh, page_size,
        num_pages, scale, chunk, window, keep, attn_scale, floor_scale, sink, slopes, softcap, status);
  }));
  JLX_LAUNCH_CHECK("attention_generic");
  return 0;
}

// ------------------------------------------------------------------------------------------------ float32, tiles of queries
// The same attention over float32 pages for head sizes that are multiples of 4 up to 128, for work items (first token row,
// count) of one request each: up to 16 tokens of a prompt portion, or one decoded token.  A block serves an item and a KV
// head: 16 RI rows, a row being a (token, query head of the group) pair, share each key tile; more rows take more blocks.
// Scores, softmax and sums as above (32-bit FMAs, two per instruction; every row's maximum and sum over its own keys).  A key
// of the tile that a row does not see has the weight -1, and its value is left out of the row's sum whatever it is (zero
// times an infinite value would not be zero); only the tiles at the rows' edges look for such weights.
// A thread has the rows ty + 16 i and of a key tile the keys tx + 16 j, then 8 columns of the output.  Keys and values come
// by asynchronous copies, the values while the scores are made; the weights lie where the keys were.
// A row's keys fall into ranges of 256 positions; each has a maximum, a sum and an output of its own, and they are merged in
// ascending order.  Where the items are few (decoding), blocks take a few ranges each and a second kernel does the merging,
// by the same operations: a row's result is a function of its position and its keys alone, however a prompt was cut.
// Bound by shared-memory reads and the FMA pipe: 1024 tokens of 16 query and 4 KV heads of 128 take 281 us (8.6 GFLOP; the
// kernel above, a block per token and KV head: 1845 us).  Contexts of a few keys would be the kernel above's (16 tokens of 16 and 4
// heads 23 us here, 13 there; 64 tokens at position 30 of 40 and 8 heads 27 and 23): they stay here, so that a position has one
// order of sums whatever it is computed with.
#define A32_KEYS 64
#define A32_RANGE 256
#define A32_TILE_TOKENS 16

struct A32Params {
  const float* q;
  const float* pages;
  const int* block_table;
  int bt_stride;
  const int* req_of_token;
  const int* positions;
  float* out;
  const int* items;  // (first token row, count) pairs; null: item i is token row rows[i], or i
  const int* rows;
  int Hq, Hkv, dh, page_size, num_pages;
  float scale;
  int chunk, window, keep;
  float attn_scale, floor_scale;
  const float* sink;
  const float* slopes;
  float softcap;
  int splits, per_split;  // blocks that share an item's ranges (1: one block merges them itself), and the ranges of one
  int part_rows;          // rows of the partial results: 0: a token's row of the step, else item * part_rows + its place in the item
  float* part_o;          // [row][Hq][splits * per_split][dh]
  float* part_ml;         // [row][Hq][splits * per_split][2]
  int* status;
};

__device__ __forceinline__ unsigned long long a32_fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
  unsigned long long d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ unsigned long long a32_mul2(unsigned long long a, unsigned long long b) {
  unsigned long long d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ unsigned long long a32_twice(float x) {
  return (unsigned long long)__float_as_uint(x) | ((unsigned long long)__float_as_uint(x) << 32);
}
__device__ __forceinline__ float a32_low(unsigned long long p) { return __uint_as_float((unsigned)p); }
__device__ __forceinline__ float a32_high(unsigned long long p) { return __uint_as_float((unsigned)(p >> 32)); }

__device__ __forceinline__ void a32_item(const A32Params& P, int item, int& n0, int& cnt) {
  if (P.items) {
    n0 = P.items[2 * item];
    cnt = P.items[2 * item + 1];
  } else {
    n0 = P.rows ? P.rows[item] : item;
    cnt = 1;
  }
}

// The ranges of an item with the positions [p_first, p_last]: those of the kept first keys, then those from the first key on
// that its first token sees; the key tiles between the two are left out.
struct A32Ranges {
  int lowest, kept_end, begin, n_kept, first_main, count;
  __device__ __forceinline__ int range(int i) const { return i < n_kept ? i : first_main + i - n_kept; }
};
__device__ __forceinline__ int a32_first_key(const A32Params& P, int p) {
  int s = P.chunk > 0 ? p / P.chunk * P.chunk : 0;
  if (P.window > 0) s = max(s, p - P.window + 1);
  return s;
}
__device__ __forceinline__ A32Ranges a32_ranges(const A32Params& P, int p_first, int p_last) {
  A32Ranges r;
  r.lowest = a32_first_key(P, p_first);
  const int kept = min(P.keep, a32_first_key(P, p_last));
  r.kept_end = (kept + A32_KEYS - 1) / A32_KEYS * A32_KEYS;
  r.begin = max(r.lowest / A32_KEYS * A32_KEYS, r.kept_end);
  r.n_kept = (r.kept_end + A32_RANGE - 1) / A32_RANGE;
  r.first_main = max(r.begin / A32_RANGE, r.n_kept);
  r.count = r.n_kept + max(0, p_last / A32_RANGE - r.first_main + 1);
  return r;
}
// (m, l, o) <- the same over two sets of keys, the second after the first.  (a: of the first, b: of the second)
__device__ __forceinline__ float a32_weights(float m_first, float m_second, float& a, float& b) {
  const float m = fmaxf(m_first, m_second);
  a = expf(m_first - m);
  b = expf(m_second - m);
  return m;
}

template <int DH, int RI>
__global__ void __launch_bounds__(256, RI == 1 ? 3 : 1) attention_f32_kernel(const __grid_constant__ A32Params P) {
  JLX_TL(TL_ATTN_GENERIC);
  constexpr int ROWS = 16 * RI, LDQ = DH + 4, LDP = A32_KEYS + 4, DV = DH / 64;
  extern __shared__ __align__(16) float smem[];
  float* Qs = smem;                  // [ROWS][LDQ]
  float* Ks = Qs + ROWS * LDQ;       // [A32_KEYS][LDQ]; then the weights [ROWS][LDP]
  float* Vs = Ks + A32_KEYS * LDQ;   // [A32_KEYS][DH]
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  const int G = P.Hq / P.Hkv, hk = blockIdx.y, dh = P.dh;
  int n0, cnt;
  a32_item(P, blockIdx.x, n0, cnt);
  const int split = blockIdx.z % P.splits, row0 = blockIdx.z / P.splits * ROWS;
  if (row0 >= cnt * G) return;
  const int p_first = P.positions[n0], p_last = p_first + cnt - 1, r = P.req_of_token[n0];
  const int start_last = a32_first_key(P, p_last);
  const A32Ranges ranges = a32_ranges(P, p_first, p_last);
  const int i_first = split * P.per_split, i_end = P.splits == 1 ? ranges.count : min(ranges.count, i_first + P.per_split);
  if (i_first >= i_end) return;
  for (int idx = tid; idx < ROWS * (DH / 4); idx += 256) {
    const int rr = idx / (DH / 4), d = idx % (DH / 4) * 4, row = row0 + rr;
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (row < cnt * G && d < dh) v = *reinterpret_cast<const float4*>(P.q + ((size_t)(n0 + row / G) * P.Hq + hk * G + row % G) * dh + d);
    *reinterpret_cast<float4*>(Qs + rr * LDQ + d) = v;
  }
  int pos[RI], start[RI];
  float qs[RI], slope[RI], m[RI], l[RI], all_m[RI], all_l[RI];
  unsigned long long acc[RI][2 * DV], all[RI][2 * DV];
#pragma unroll
  for (int i = 0; i < RI; ++i) {
    const int row = row0 + ty + 16 * i;
    const bool there = row < cnt * G;
    pos[i] = there ? p_first + row / G : -1;  // -1: sees no key
    start[i] = there ? a32_first_key(P, pos[i]) : 0;
    qs[i] = P.scale;
    if (P.attn_scale != 0.f && there) qs[i] *= 1.f + P.attn_scale * log1pf(floorf(((float)pos[i] + 1.f) / P.floor_scale));
    slope[i] = P.slopes && there ? P.slopes[hk * G + row % G] : 0.f;
    all_m[i] = -INFINITY;
    all_l[i] = 0.f;
#pragma unroll
    for (int c = 0; c < 2 * DV; ++c) all[i][c] = 0ull;
  }
  const size_t page_elems = (size_t)2 * P.Hkv * P.page_size * dh;
  auto copy_rows = [&](int t0, int end, float* dst, int ld, int plane) {
    for (int idx = tid; idx < A32_KEYS * (DH / 4); idx += 256) {
      const int j = idx / (DH / 4), d = idx % (DH / 4) * 4, at = t0 + j;
      const float* src = P.pages;
      bool there = at < end && (at >= ranges.lowest || at < P.keep) && d < dh;  // pages of other keys may have been given back
      if (there) {
        const int page = P.block_table[(size_t)r * P.bt_stride + at / P.page_size];
        if (page < 0 || page >= P.num_pages) {
          atomicOr(P.status, JLX_STATUS_BAD_PAGE);
          there = false;
        } else {
          src = P.pages + (size_t)page * page_elems + ((size_t)(plane * P.Hkv + hk) * P.page_size + at % P.page_size) * dh + d;
        }
      }
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((unsigned)__cvta_generic_to_shared(dst + j * ld + d)), "l"(src),
                   "r"(there ? 16 : 0) : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  for (int ri = i_first; ri < i_end; ++ri) {
#pragma unroll
    for (int i = 0; i < RI; ++i) {
      m[i] = -INFINITY;
      l[i] = 0.f;
#pragma unroll
      for (int c = 0; c < 2 * DV; ++c) acc[i][c] = 0ull;
    }
    const int range0 = ranges.range(ri) * A32_RANGE, end = min(p_last + 1, range0 + A32_RANGE);
    for (int t0 = range0; t0 < end; t0 += A32_KEYS) {
      if (t0 >= ranges.kept_end && t0 < ranges.begin) continue;
      __syncthreads();  // the tile before is consumed; the queries are there
      copy_rows(t0, end, Ks, LDQ, 0);
      copy_rows(t0, end, Vs, DH, 1);
      asm volatile("cp.async.wait_group 1;" ::: "memory");
      __syncthreads();
      unsigned long long s2[RI][4];
#pragma unroll
      for (int i = 0; i < RI; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) s2[i][j] = 0ull;
#pragma unroll 4
      for (int d = 0; d < DH; d += 4) {
        ulonglong2 k[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) k[j] = *reinterpret_cast<const ulonglong2*>(Ks + (tx + 16 * j) * LDQ + d);
#pragma unroll
        for (int i = 0; i < RI; ++i) {
          const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(Qs + (ty + 16 * i) * LDQ + d);
#pragma unroll
          for (int j = 0; j < 4; ++j) s2[i][j] = a32_fma2(a.y, k[j].y, a32_fma2(a.x, k[j].x, s2[i][j]));
        }
      }
      __syncthreads();  // the keys are read: the weights take their place
#pragma unroll
      for (int i = 0; i < RI; ++i) {
        float s[4], top = -INFINITY;
        bool seen[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int at = t0 + tx + 16 * j;
          float x = (a32_low(s2[i][j]) + a32_high(s2[i][j])) * qs[i];
          if (P.softcap > 0.f) x = P.softcap * tanhf(x / P.softcap);
          x = fmaf(-slope[i], (float)(pos[i] - at), x);
          seen[j] = at < end && at <= pos[i] && (at >= start[i] || at < P.keep);
          s[j] = seen[j] ? x : -INFINITY;
          top = fmaxf(top, s[j]);
        }
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
        const float m_new = fmaxf(m[i], top);
        const float base = m_new == -INFINITY ? 0.f : m_new;  // no key so far: all weights are zero
        const float corr = expf(m[i] - base);
        float sum = 0.f;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float w = expf(s[j] - base);
          Ks[(ty + 16 * i) * LDP + tx + 16 * j] = seen[j] ? w : -1.f;
          sum += w;
        }
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
        l[i] = l[i] * corr + sum;
        m[i] = m_new;
        const unsigned long long c2 = a32_twice(corr);
#pragma unroll
        for (int c = 0; c < 2 * DV; ++c) acc[i][c] = a32_mul2(acc[i][c], c2);
      }
      asm volatile("cp.async.wait_group 0;" ::: "memory");
      __syncthreads();  // weights and values are there
      auto add_values = [&](auto all_seen) {
#pragma unroll 2
        for (int j = 0; j < A32_KEYS; j += 4) {
          float4 w[RI];
#pragma unroll
          for (int i = 0; i < RI; ++i) w[i] = *reinterpret_cast<const float4*>(Ks + (ty + 16 * i) * LDP + j);
#pragma unroll
          for (int jj = 0; jj < 4; ++jj)
#pragma unroll
            for (int h = 0; h < DV; ++h) {
              const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(Vs + (j + jj) * DH + 64 * h + 4 * tx);
#pragma unroll
              for (int i = 0; i < RI; ++i) {
                const float wj = jj == 0 ? w[i].x : (jj == 1 ? w[i].y : (jj == 2 ? w[i].z : w[i].w));
                if (!decltype(all_seen)::value && wj < 0.f) continue;
                const unsigned long long x = a32_twice(wj);
                acc[i][2 * h] = a32_fma2(x, v.x, acc[i][2 * h]);
                acc[i][2 * h + 1] = a32_fma2(x, v.y, acc[i][2 * h + 1]);
              }
            }
        }
      };
      // (rows that are not there: whatever they add is not stored)
      if (t0 + A32_KEYS - 1 <= p_first && (t0 >= start_last || t0 + A32_KEYS <= P.keep)) add_values(std::true_type());
      else add_values(std::false_type());
    }
#pragma unroll
    for (int i = 0; i < RI; ++i) {
      const int row = row0 + ty + 16 * i;
      if (P.splits > 1) {
        if (row >= cnt * G) continue;
        const int part_row = P.part_rows ? blockIdx.x * P.part_rows + row / G : n0 + row / G;
        const size_t at = ((size_t)part_row * P.Hq + hk * G + row % G) * (P.splits * P.per_split) + ri;
        if (tx == 0) {
          P.part_ml[2 * at] = m[i];
          P.part_ml[2 * at + 1] = l[i];
        }
#pragma unroll
        for (int h = 0; h < DV; ++h) {
          const int d = 64 * h + 4 * tx;
          if (d < dh)
            *reinterpret_cast<float4*>(P.part_o + at * dh + d) =
                make_float4(a32_low(acc[i][2 * h]), a32_high(acc[i][2 * h]), a32_low(acc[i][2 * h + 1]), a32_high(acc[i][2 * h + 1]));
        }
      } else if (l[i] != 0.f) {  // else a range without a key that the row sees
        float a, b;
        all_m[i] = a32_weights(all_m[i], m[i], a, b);
        all_l[i] = fmaf(l[i], b, all_l[i] * a);
#pragma unroll
        for (int c = 0; c < 2 * DV; ++c) all[i][c] = a32_fma2(acc[i][c], a32_twice(b), a32_mul2(all[i][c], a32_twice(a)));
      }
    }
  }
  if (P.splits > 1) return;
#pragma unroll
  for (int i = 0; i < RI; ++i) {
    const int row = row0 + ty + 16 * i;
    if (row >= cnt * G) continue;
    const int n = n0 + row / G, h = hk * G + row % G;
    float by = 1.f, sum = all_l[i];
    if (P.sink) {  // the sink joins the sum like a last key without a value
      float b;
      a32_weights(all_m[i], P.sink[h], by, b);
      sum = fmaf(1.f, b, sum * by);
    }
    float* dst = P.out + ((size_t)n * P.Hq + h) * dh;
#pragma unroll
    for (int hh = 0; hh < DV; ++hh) {
      const int d = 64 * hh + 4 * tx;
      if (d < dh)
        *reinterpret_cast<float4*>(dst + d) = make_float4(a32_low(all[i][2 * hh]) * by / sum, a32_high(all[i][2 * hh]) * by / sum,
                                                          a32_low(all[i][2 * hh + 1]) * by / sum, a32_high(all[i][2 * hh + 1]) * by / sum);
    }
  }
}

// Merges the ranges of every row of an item, as the kernel above does where one block has them all: one warp per (token, head).
__global__ void __launch_bounds__(128) attention_f32_combine_kernel(const __grid_constant__ A32Params P, int max_count) {
  JLX_TL(TL_ATTN_COMBINE);
  int n0, cnt;
  a32_item(P, blockIdx.x / max_count, n0, cnt);
  const int t = blockIdx.x % max_count, lane = threadIdx.x & 31, h = blockIdx.y * 4 + (threadIdx.x >> 5);
  if (t >= cnt || h >= P.Hq) return;
  const int p_first = P.positions[n0], count = min(a32_ranges(P, p_first, p_first + cnt - 1).count, P.splits * P.per_split);
  const size_t at = ((size_t)(P.part_rows ? blockIdx.x : n0 + t) * P.Hq + h) * (P.splits * P.per_split);
  float all_m = -INFINITY, all_l = 0.f;
  float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
  const int d = 4 * lane;
#pragma unroll 4
  for (int s = 0; s < count; ++s) {
    const float m = P.part_ml[2 * (at + s)], l = P.part_ml[2 * (at + s) + 1];
    const float4 v = d < P.dh ? *reinterpret_cast<const float4*>(P.part_o + (at + s) * P.dh + d) : make_float4(0.f, 0.f, 0.f, 0.f);
    if (l == 0.f) continue;
    float a, b;
    all_m = a32_weights(all_m, m, a, b);
    all_l = fmaf(l, b, all_l * a);
    o = make_float4(fmaf(v.x, b, o.x * a), fmaf(v.y, b, o.y * a), fmaf(v.z, b, o.z * a), fmaf(v.w, b, o.w * a));
  }
  float by = 1.f;
  if (P.sink) {
    float b;
    a32_weights(all_m, P.sink[h], by, b);
    all_l = fmaf(1.f, b, all_l * by);
  }
  if (d < P.dh)
    *reinterpret_cast<float4*>(P.out + ((size_t)(n0 + t) * P.Hq + h) * P.dh + d) =
        make_float4(o.x * by / all_l, o.y * by / all_l, o.z * by / all_l, o.w * by / all_l);
}

JLX_API int jlx_attention_f32_supported(int dh) { return dh > 0 && dh % 4 == 0 && dh <= 128; }

template <int DH, int RI>
static cudaError_t launch_attention_f32(const A32Params& P, int n_items, int row_blocks, cudaStream_t stream) {
  const size_t smem = sizeof(float) * ((size_t)16 * RI * (DH + 4) + (size_t)A32_KEYS * (DH + 4) + (size_t)A32_KEYS * DH);
  const cudaError_t e = cudaFuncSetAttribute(attention_f32_kernel<DH, RI>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  attention_f32_kernel<DH, RI><<<dim3(n_items, P.Hkv, row_blocks * P.splits), 256, smem, stream>>>(P);
  return cudaGetLastError();
}

// n_items items of at most max_count tokens (items null: single tokens, rows[i] or i).  part_o, part_ml: for splits > 1, room for
// every token row of the step, or (part_by_item) for n_items * max_count rows.
JLX_API int jlx_attention_f32(const float* q, const float* pages, const int* block_table, int bt_stride, const int* req_of_token,
                              const int* positions, float* out, int Hq, int Hkv, int dh, int page_size, int num_pages, float scale,
                              int chunk, int window, int keep, float attn_scale, float floor_scale, const float* sink, const float* slopes,
                              float softcap, const int* items, const int* rows, int n_items, int max_count, int splits, int per_split,
                              int part_by_item, float* part_o, float* part_ml, int* status, cudaStream_t stream) {
  JLX_REQUIRE(Hq > 0 && Hkv > 0 && page_size > 0 && num_pages > 0 && n_items >= 0, "attention_f32: bad sizes");
  JLX_REQUIRE(Hq % Hkv == 0 && Hkv <= 65535, "attention_f32: %d query heads for %d KV heads", Hq, Hkv);
  JLX_REQUIRE(jlx_attention_f32_supported(dh), "attention_f32: head size %d is no multiple of 4 up to 128", dh);
  JLX_REQUIRE((((uintptr_t)q | (uintptr_t)pages | (uintptr_t)out) & 15) == 0, "attention_f32: rows must start on 16-byte boundaries");
  JLX_REQUIRE(softcap >= 0.f && keep >= 0 && (attn_scale == 0.f || floor_scale > 0.f), "attention_f32: bad score cap, kept keys or floor_scale");
  JLX_REQUIRE(max_count >= 1 && max_count <= A32_TILE_TOKENS && (items || max_count == 1), "attention_f32: items of up to %d tokens", A32_TILE_TOKENS);
  JLX_REQUIRE(splits >= 1 && (splits == 1 || (per_split > 0 && part_o && part_ml)), "attention_f32: bad key ranges");
  if (n_items == 0) return 0;
  const int rows_of_item = max_count * (Hq / Hkv);
  const bool few = rows_of_item <= 16;
  const int row_blocks = (rows_of_item + (few ? 15 : 63)) / (few ? 16 : 64);
  JLX_REQUIRE((long long)row_blocks * splits <= 65535, "attention_f32: too many key ranges");
  const A32Params P = {q, pages, block_table, bt_stride, req_of_token, positions, out, items, rows, Hq, Hkv, dh, page_size, num_pages, scale,
                       chunk, window, keep, attn_scale, floor_scale, sink, slopes, softcap, splits, per_split, part_by_item ? max_count : 0, part_o,
                       part_ml, status};
  if (dh <= 64) JLX_CUDA((few ? launch_attention_f32<64, 1>(P, n_items, row_blocks, stream) : launch_attention_f32<64, 4>(P, n_items, row_blocks, stream)));
  else JLX_CUDA((few ? launch_attention_f32<128, 1>(P, n_items, row_blocks, stream) : launch_attention_f32<128, 4>(P, n_items, row_blocks, stream)));
  if (splits > 1) {
    attention_f32_combine_kernel<<<dim3(n_items * max_count, (Hq + 3) / 4), 128, 0, stream>>>(P, max_count);
    JLX_LAUNCH_CHECK("attention_f32_combine");
  }
  return 0;
}

// The difference of two maps (see attention_maps.cuh) as a kernel of its own, behind the kernel above: attn float32
// [N, 2 H, dpad] -> out rows.  One warp per (token, head).
template <typename TO>
__global__ void map_difference_kernel(const float* __restrict__ attn, TO* __restrict__ out, MapDifference D, int items, int H, int dpad) {
  JLX_TL(TL_OTHER);
  pdl_launch_dependents_if_small();
  pdl_wait();
  const int lane = threadIdx.x & 31;
  const int item = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (item >= items) return;
  const int n = item / H, h = item - n * H;
  const float* a1 = attn + (size_t)item * 2 * dpad;
  const float* a2 = a1 + dpad;
  float ss = 0.f;
  for (int c = lane; c < D.out_dim; c += 32) {
    const float o = a1[c] - D.weight * a2[c];
    ss = fmaf(o, o, ss);
  }
  const float rms = sqrtf(warp_sum(ss) / (float)D.out_dim + D.eps);
  TO* dst = out + (size_t)n * D.ld_out + (size_t)h * D.out_dim;
  for (int c = lane; c < D.out_dim; c += 32) dst[c] = from_f32<TO>((a1[c] - D.weight * a2[c]) / rms * D.mult);
}

JLX_API int jlx_map_difference(const float* attn, void* out, int out_dtype, const MapDifference* diff, int N, int H, int dpad,
                               cudaStream_t stream) {
  JLX_REQUIRE(N >= 0 && H > 0 && diff && diff->out_dim > 0 && dpad >= diff->out_dim, "map_difference: bad sizes");
  if (N == 0) return 0;
  JLX_REQUIRE((long long)N * H < (1ll << 31), "map_difference: too many heads");
  const int items = N * H;
  JLX_DISPATCH_DTYPE(out_dtype, TO, {
    JLX_CUDA(jlx_launch_pdl(map_difference_kernel<TO>, dim3((items + 3) / 4), dim3(128), 0, stream, attn, (TO*)out, *diff, items, H, dpad));
  });
  JLX_LAUNCH_CHECK("map_difference");
  return 0;
}
