// Next-token choice from 32-bit logits: argmax, or temperature sampling over the k most likely
// tokens (all of them when k = 0) with a counter-based random number per request.
//
// Reference: llama4 decodes by argmax only (llama4/llama4_jax/model.py:1266,1275).  The repository's
// sampler is gpt_oss/gpt_oss_jax/model.py:1125-1147: softmax(logits / temp), top-k, normalised
// cumulative sum, first index whose cumulative probability reaches the uniform draw; temp <= 1e-3
// means argmax.  The draw here is Philox-4x32-10 keyed by (seed, request stream) with the request's
// step as counter, so a request's tokens do not depend on what else is in the batch.
#include "common.cuh"
#include "sampling_noalloc.h"

#define SAMPLE_MAX_K 64

__device__ __forceinline__ void philox4x32_10(uint32_t c[4], uint32_t k0, uint32_t k1) {
  const uint32_t M0 = 0xD2511F53u, M1 = 0xCD9E8D57u, W0 = 0x9E3779B9u, W1 = 0xBB67AE85u;
#pragma unroll
  for (int r = 0; r < 10; ++r) {
    const uint32_t hi0 = __umulhi(M0, c[0]), lo0 = M0 * c[0];
    const uint32_t hi1 = __umulhi(M1, c[2]), lo1 = M1 * c[2];
    const uint32_t n0 = hi1 ^ c[1] ^ k0, n1 = lo1, n2 = hi0 ^ c[3] ^ k1, n3 = lo0;
    c[0] = n0; c[1] = n1; c[2] = n2; c[3] = n3;
    k0 += W0; k1 += W1;
  }
}

struct ArgMax {
  float v;
  int i;
};

__device__ __forceinline__ ArgMax better(ArgMax a, ArgMax b) {
  // larger value wins; equal values: lower index wins; index -1 = empty
  if (b.i < 0) return a;
  if (a.i < 0) return b;
  if (b.v > a.v || (b.v == a.v && b.i < a.i)) return b;
  return a;
}

__device__ ArgMax block_argmax(ArgMax a, ArgMax* scratch) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    ArgMax b;
    b.v = __shfl_xor_sync(0xffffffffu, a.v, o);
    b.i = __shfl_xor_sync(0xffffffffu, a.i, o);
    a = better(a, b);
  }
  __syncthreads();
  if (lane == 0) scratch[warp] = a;
  __syncthreads();
  if (warp == 0) {
    ArgMax t = lane < nwarp ? scratch[lane] : ArgMax{0.f, -1};
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      ArgMax b;
      b.v = __shfl_xor_sync(0xffffffffu, t.v, o);
      b.i = __shfl_xor_sync(0xffffffffu, t.i, o);
      t = better(t, b);
    }
    if (lane == 0) scratch[32] = t;
  }
  __syncthreads();
  return scratch[32];
}

// ---- sampling in three launches.  A row's logits are read once, by several blocks:
//
//   sample_top_kernel     (row, chunk): the chunk's `k` largest (value, index), in no order; one for rows that need only
//                         their largest (greedy rows, and rows that draw from the whole vocabulary).
//   sample_spans_kernel   (row, spans): for rows that draw from the whole vocabulary, the sums of exp over SAMPLE_SPANS
//                         contiguous spans of the row; blocks of other rows leave at once.
//   sample_pick_kernel    (row): the chunks' lists merged, the draw, the choice.
//
// What bounds it: the one pass over the logits (64 rows x 202048: 52 MB, 8 us at the copy rate), then the latency of three
// dependent launches and of the counts that find the k-th largest.  The kernel that was here walked a row once per chosen
// token in one block: 64 rows, top 64: 3630 us; these three: 48 us (greedy rows 24 us, the whole vocabulary 93 us: the
// sums of the spans, a sequential prefix over them and one over the chosen span).
// Every sum runs in the order it had there (the chosen tokens in descending order; the spans each in index order, then
// the tree over the spans), so the drawn tokens are the same.
#define SAMPLE_THREADS 512        // of sample_top_kernel: a block's threads, and so the strands it cuts a chunk into
#define SAMPLE_STRAND 64          // values that one thread reads at most
#define SAMPLE_MAX_CANDIDATES (SAMPLE_MAX_K * SAMPLE_STRAND)
#define SAMPLE_SPANS 1024
#define SAMPLE_SPANS_PER_BLOCK 64
#define SAMPLE_PIECE 64           // values of each span that a block holds at once

// (value, index) as one number: larger values first, equal values by the lower index; 0: no entry (no number maps there).
typedef unsigned long long SampleKey;
__device__ __forceinline__ unsigned sample_order(float v) {  // 0 for what is not a number; -0 counts as +0
  const unsigned u = __float_as_uint(v + 0.f);
  return isnan(v) ? 0u : ((u & 0x80000000u) ? ~u : (u | 0x80000000u));
}
__device__ __forceinline__ SampleKey sample_key(unsigned order, int i) {
  return order == 0u ? 0ull : ((SampleKey)order << 32) | (unsigned)(0xffffffffu - (unsigned)i);
}
__device__ __forceinline__ float sample_value(SampleKey k) {
  const unsigned o = (unsigned)(k >> 32);
  return __uint_as_float((o & 0x80000000u) ? (o & 0x7fffffffu) : ~o);
}
__device__ __forceinline__ int sample_index(SampleKey k) { return (int)(0xffffffffu - (unsigned)k); }

// Sorts n keys (a power of two) in shared memory, largest first; all threads of the block call it.
__device__ __forceinline__ void sample_sort(SampleKey* a, int n) {
  for (int size = 2; size <= n; size <<= 1)
    for (int step = size >> 1; step > 0; step >>= 1) {
      __syncthreads();
      for (int t = threadIdx.x; t < (n >> 1); t += blockDim.x) {
        const int i = 2 * t - (t & (step - 1)), j = i + step;
        const SampleKey x = a[i], y = a[j];
        if (((i & size) == 0) == (x < y)) {
          a[i] = y;
          a[j] = x;
        }
      }
    }
  __syncthreads();
}

__device__ __forceinline__ int sample_pow2(int n) {
  int p = 2;
  while (p < n) p <<= 1;
  return p;
}

// The candidates a row's draw chooses among: its largest alone, all (0), or the k largest.
__device__ __forceinline__ int sample_k(const float* temperature, const int* top_k, int m, int V) {
  if (!temperature || temperature[m] <= 1e-3f) return 1;
  const int k = top_k ? top_k[m] : 0;
  return k <= 0 ? 0 : min(min(k, V), SAMPLE_MAX_K);  // the host refuses larger k before the launch
}

// The largest key `from` that at least k of the block's keys (one per thread, all different or 0) reach: bit by bit, each
// bit one count over the block, until exactly k reach it (a dozen or two bits; a sort of the 512 keys was a third of the
// kernel).  Fewer than k keys that are not 0: 1.
__device__ __forceinline__ SampleKey sample_kth(SampleKey mine, int k) {
  SampleKey from = 0ull;
  if (__syncthreads_count(mine != 0ull) <= k) return 1ull;
  for (int bit = 63; bit >= 0; --bit) {
    const SampleKey t = from | (1ull << bit);
    const int reach = __syncthreads_count(mine >= t);
    if (reach >= k) from = t;
    if (reach == k) break;
  }
  return from;
}

// A chunk's k largest, in no order: every thread finds the largest of its strand; a value among the chunk's k largest lies
// in a strand whose largest is among the k largest of those, so only these k threads read their strand again (at most
// SAMPLE_STRAND values each: the list of candidates cannot overflow) and keep what reaches the k-th strand's largest.
__global__ void __launch_bounds__(SAMPLE_THREADS, 4)  // 64 rows of 202048 are 512 blocks: all resident at once
sample_top_kernel(const float* __restrict__ logits, int V, long long ld, int chunk, const float* __restrict__ temperature,
                  const int* __restrict__ top_k, SampleKey* __restrict__ lists) {
  JLX_TL(TL_SAMPLE);
  __shared__ SampleKey keys[SAMPLE_MAX_CANDIDATES];
  __shared__ int count, kept;
  const int m = blockIdx.x, tid = threadIdx.x;
  pdl_launch_dependents();
  pdl_wait();
  const int k = max(1, sample_k(temperature, top_k, m, V));
  const float* row = logits + (size_t)m * ld;
  const int lo = blockIdx.y * chunk, hi = min(V, lo + chunk);
  SampleKey* list = lists + ((size_t)m * gridDim.y + blockIdx.y) * SAMPLE_MAX_K;
  // one strand: every SAMPLE_THREADS-th group of four values, then every SAMPLE_THREADS-th of the rest; AHEAD groups are
  // in flight together
  float best = -INFINITY;
  int at = -1;
  const bool vec = (ld & 3) == 0 && ((uintptr_t)logits & 15) == 0;  // chunks are multiples of 4
  const int hi4 = vec ? lo + ((hi - lo) & ~3) : lo;
  constexpr int AHEAD = 4, STEP = 4 * SAMPLE_THREADS;
  for (int i0 = lo + 4 * tid; i0 < hi4; i0 += AHEAD * STEP) {
    float4 v[AHEAD];
#pragma unroll
    for (int g = 0; g < AHEAD; ++g)
      v[g] = i0 + g * STEP < hi4 ? *reinterpret_cast<const float4*>(row + i0 + g * STEP) : make_float4(-INFINITY, -INFINITY, -INFINITY, -INFINITY);
#pragma unroll
    for (int g = 0; g < AHEAD; ++g) {
      const int i = i0 + g * STEP;
      if (v[g].x > best) { best = v[g].x; at = i; }
      if (v[g].y > best) { best = v[g].y; at = i + 1; }
      if (v[g].z > best) { best = v[g].z; at = i + 2; }
      if (v[g].w > best) { best = v[g].w; at = i + 3; }
    }
  }
#pragma unroll 4
  for (int i = hi4 + tid; i < hi; i += SAMPLE_THREADS) {
    const float v = row[i];
    if (v > best) { best = v; at = i; }
  }
  if (at < 0) {  // nothing above minus infinity: its first place, if the strand has one
    for (int i = lo + 4 * tid; i < hi4 && at < 0; i += STEP)
      for (int c = 3; c >= 0; --c)
        if (!isnan(row[i + c])) at = i + c;
    for (int i = hi4 + tid; i < hi && at < 0; i += SAMPLE_THREADS)
      if (!isnan(row[i])) at = i;
  }
  const SampleKey mine = at < 0 ? 0ull : sample_key(sample_order(best), at);
  if (k == 1) {
    SampleKey w = mine;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const SampleKey x = __shfl_xor_sync(0xffffffffu, w, o);
      w = x > w ? x : w;
    }
    if ((tid & 31) == 0) keys[tid >> 5] = w;
    __syncthreads();
    if (tid == 0) {
      for (int i = 1; i < SAMPLE_THREADS / 32; ++i) w = keys[i] > w ? keys[i] : w;
      list[0] = w;
    }
    return;
  }
  const SampleKey from = sample_kth(mine, k);
  if (tid == 0) count = kept = 0;
  __syncthreads();
  if (mine >= from) {
    for (int i0 = lo + 4 * tid; i0 < hi4; i0 += AHEAD * STEP) {
      float4 v[AHEAD];
#pragma unroll
      for (int g = 0; g < AHEAD; ++g)
        v[g] = i0 + g * STEP < hi4 ? *reinterpret_cast<const float4*>(row + i0 + g * STEP) : make_float4(NAN, NAN, NAN, NAN);
#pragma unroll
      for (int g = 0; g < AHEAD; ++g) {
        const float vv[4] = {v[g].x, v[g].y, v[g].z, v[g].w};
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const SampleKey x = sample_key(sample_order(vv[c]), i0 + g * STEP + c);
          if (x >= from) keys[atomicAdd(&count, 1)] = x;
        }
      }
    }
    for (int i = hi4 + tid; i < hi; i += SAMPLE_THREADS) {
      const SampleKey x = sample_key(sample_order(row[i]), i);
      if (x >= from) keys[atomicAdd(&count, 1)] = x;
    }
  }
  __syncthreads();
  const int n = count;
  if (n > SAMPLE_THREADS) {  // many large values in few strands
    const int p = sample_pow2(n);
    for (int i = n + tid; i < p; i += SAMPLE_THREADS) keys[i] = 0ull;
    sample_sort(keys, p);
    if (tid < k) list[tid] = keys[tid];
    return;
  }
  const SampleKey x = tid < n ? keys[tid] : 0ull;
  const SampleKey reach = sample_kth(x, k);
  if (x >= reach) list[atomicAdd(&kept, 1)] = x;
  __syncthreads();
  if (tid >= kept && tid < k) list[tid] = 0ull;
}

// The largest entry of a row whose chunks list only theirs; every thread gets it.
__device__ __forceinline__ SampleKey sample_best(const SampleKey* lists, int m, int chunks) {
  SampleKey w = 0ull;
  for (int c = threadIdx.x & 31; c < chunks; c += 32) {
    const SampleKey x = lists[((size_t)m * chunks + c) * SAMPLE_MAX_K];
    w = x > w ? x : w;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const SampleKey x = __shfl_xor_sync(0xffffffffu, w, o);
    w = x > w ? x : w;
  }
  return w;
}

__global__ void __launch_bounds__(256)
sample_spans_kernel(const float* __restrict__ logits, int V, long long ld, int chunks, const float* __restrict__ temperature,
                    const int* __restrict__ top_k, const SampleKey* __restrict__ lists, float* __restrict__ sums) {
  JLX_TL(TL_SAMPLE);
  __shared__ float piece[SAMPLE_SPANS_PER_BLOCK][SAMPLE_PIECE + 1];
  const int m = blockIdx.x, tid = threadIdx.x;
  pdl_launch_dependents();
  pdl_wait();
  if (sample_k(temperature, top_k, m, V) != 0) return;
  const SampleKey best = sample_best(lists, m, chunks);
  if (best == 0ull) return;
  const float mx = sample_value(best), inv_t = 1.f / temperature[m];
  const float* row = logits + (size_t)m * ld;
  const int span = (V + SAMPLE_SPANS - 1) / SAMPLE_SPANS, first = blockIdx.y * SAMPLE_SPANS_PER_BLOCK;
  float s = 0.f;
  for (int off = 0; off < span; off += SAMPLE_PIECE) {
    const int width = min(SAMPLE_PIECE, span - off);
    __syncthreads();
    for (int idx = tid; idx < SAMPLE_SPANS_PER_BLOCK * SAMPLE_PIECE; idx += 256) {
      const int t = idx / SAMPLE_PIECE, i = idx % SAMPLE_PIECE;
      const long long at = (long long)(first + t) * span + off + i;
      float e = 0.f;
      if (i < width && at < V) {
        const float v = row[at];
        if (!isnan(v)) e = expf((v - mx) * inv_t);
      }
      piece[t][i] = e;
    }
    __syncthreads();
    if (tid < SAMPLE_SPANS_PER_BLOCK)
      for (int i = 0; i < width; ++i) s += piece[tid][i];
  }
  if (tid < SAMPLE_SPANS_PER_BLOCK) sums[(size_t)m * SAMPLE_SPANS + first + tid] = s;
}

// One block of SAMPLE_SPANS threads per row.  params per row: temperature[m], top_k[m], stream[m] (request's random
// stream), counter[m] (request's step).  Rows with temperature <= 1e-3 take the argmax.
__global__ void __launch_bounds__(SAMPLE_SPANS)
sample_pick_kernel(const float* __restrict__ logits, int V, long long ld, int chunks, const float* __restrict__ temperature,
                   const int* __restrict__ top_k, const unsigned long long* __restrict__ streams,
                   const unsigned long long* __restrict__ counters, unsigned long long seed,
                   const SampleKey* __restrict__ lists, const float* __restrict__ sums, int* __restrict__ out) {
  JLX_TL(TL_SAMPLE);
  __shared__ SampleKey keys[SAMPLE_MAX_K];
  __shared__ float weight[SAMPLE_SPANS], upto[SAMPLE_SPANS], fscratch[33];
  __shared__ int pick;
  const int m = blockIdx.x, tid = threadIdx.x;
  pdl_wait();
  const int want = sample_k(temperature, top_k, m, V);
  const float temp = temperature ? temperature[m] : 0.f;
  int kept = 0;
  if (want > 1) {
    // merge: the best `want` so far stay while the other lists pass by, then each finds its place by counting the larger
    const int total_keys = chunks * want;
    for (int from = 0; from < total_keys;) {
      const int take = min(SAMPLE_SPANS - kept, total_keys - from);
      const int e = from + tid - kept;
      SampleKey x = 0ull;
      if (tid < kept) x = keys[tid];
      else if (tid < kept + take) x = lists[((size_t)m * chunks + e / want) * SAMPLE_MAX_K + e % want];
      const SampleKey reach = sample_kth(x, want);
      if (tid == 0) pick = 0;
      __syncthreads();
      if (x >= reach) keys[atomicAdd(&pick, 1)] = x;
      __syncthreads();
      kept = pick;
      from += take;
      __syncthreads();
    }
    const SampleKey x = tid < kept ? keys[tid] : 0ull;
    int place = 0;
    if (tid < kept)
      for (int j = 0; j < kept; ++j) place += keys[j] > x;
    __syncthreads();
    if (tid < kept) keys[place] = x;
    if (tid == 0 && kept == 0) keys[0] = 0ull;
    __syncthreads();
  }
  const SampleKey best = want > 1 ? keys[0] : sample_best(lists, m, chunks);
  if (want == 1 || best == 0ull) {  // greedy, or the one candidate
    if (tid == 0) out[m] = best == 0ull ? 0 : sample_index(best);
    return;
  }
  // uniform draw for this (request stream, step)
  uint32_t c[4] = {(uint32_t)counters[m], (uint32_t)(counters[m] >> 32), (uint32_t)streams[m], (uint32_t)(streams[m] >> 32)};
  philox4x32_10(c, (uint32_t)seed, (uint32_t)(seed >> 32));
  const float u = (float)(c[0] >> 8) * (1.0f / 16777216.0f);
  const float inv_t = 1.f / temp;
  const float mx = sample_value(best);

  if (want > 0) {
    const int k = kept;  // a row may hold fewer numbers than were asked for
    if (tid < k) weight[tid] = expf((sample_value(keys[tid]) - mx) * inv_t);
    __syncthreads();
    if (tid < 32) {
      if (tid == 0) {
        float run = 0.f;
#pragma unroll 8
        for (int j = 0; j < k; ++j) {  // in descending order of the weights
          run += weight[j];
          upto[j] = run;
        }
      }
      __syncwarp();
      const float total = upto[k - 1];
      int first = k - 1;
      for (int j = tid; j < k; j += 32)
        if (u <= upto[j] / total) { first = min(first, j); break; }
      first = __reduce_min_sync(0xffffffffu, first);
      if (tid == 0) out[m] = sample_index(keys[first]);
    }
    return;
  }
  // whole vocabulary, cumulative sum in index order: thread t stands for one contiguous span
  const float* row = logits + (size_t)m * ld;
  const int span = (V + SAMPLE_SPANS - 1) / SAMPLE_SPANS;
  weight[tid] = sums[(size_t)m * SAMPLE_SPANS + tid];
  const float total = block_sum(weight[tid], fscratch);
  if (tid == 0) {
    pick = SAMPLE_SPANS - 1;
    float run = 0.f;
#pragma unroll 8
    for (int t = 0; t < SAMPLE_SPANS; ++t) {
      run += weight[t];
      upto[t] = run;
    }
  }
  __syncthreads();
  if (u <= upto[tid] / total) atomicMin(&pick, tid);
  __syncthreads();
  const int t = pick;  // the span that the draw falls into; then the index inside it
  float run = t > 0 ? upto[t - 1] : 0.f;
  const int l2 = (int)min((long long)V, (long long)t * span), h2 = min(V, l2 + span);
  __syncthreads();
  if (tid == 0) pick = V;
  __syncthreads();  // (a span behind the row's end is empty: the loop has no barrier then)
  for (int i0 = l2; i0 < h2; i0 += SAMPLE_SPANS) {
    const int i = i0 + tid, n = min(SAMPLE_SPANS, h2 - i0);
    const float v = i < h2 ? row[i] : 0.f;
    const bool number = i < h2 && !isnan(v);
    weight[tid] = number ? expf((v - mx) * inv_t) : 0.f;
    __syncthreads();
    if (tid == 0) {
      float r = run;
#pragma unroll 8
      for (int j = 0; j < n; ++j) {
        r += weight[j];
        upto[j] = r;
      }
    }
    __syncthreads();
    if (number && u <= upto[tid] / total) atomicMin(&pick, i);
    run = upto[n - 1];
    __syncthreads();
    if (pick < V) break;
  }
  if (pick >= V) {  // rounding at the very end of the range: last token with weight
    __syncthreads();
    if (tid == 0) pick = -1;
    __syncthreads();
    int last = -1;
    for (int i = tid; i < V; i += SAMPLE_SPANS)
      if (!isnan(row[i]) && expf((row[i] - mx) * inv_t) > 0.f) last = i;
    if (last >= 0) atomicMax(&pick, last);
    __syncthreads();
    if (tid == 0 && pick < 0) pick = sample_index(best);
  }
  __syncthreads();
  if (tid == 0) out[m] = pick;
}

// Greedy choice in two stages so that a handful of rows still uses the whole GPU: each block finds the
// best (value, index) of one chunk of a row; one block per row then picks among the chunks.  Ties go to
// the lower index in both stages.
#define ARGMAX_CHUNKS 32
__global__ void __launch_bounds__(256)
argmax_chunk_kernel(const float* __restrict__ logits, int V, long long ld, float* __restrict__ part_v, int* __restrict__ part_i) {
  JLX_TL(TL_ARGMAX);
  __shared__ ArgMax scratch[33];
  const int m = blockIdx.y, c = blockIdx.x;
  const int span = ((V + ARGMAX_CHUNKS - 1) / ARGMAX_CHUNKS + 3) / 4 * 4;  // a multiple of 4: chunks start 16-byte aligned
  const int lo = min(V, c * span), hi = min(V, lo + span);
  const float* row = logits + (size_t)m * ld;
  ArgMax best{0.f, -1};
  if ((ld & 3) == 0 && ((uintptr_t)logits & 15) == 0) {
    // four values per access and a thread's accesses in flight together: a step's one or few rows are read at the speed
    // of a memory latency per round, so there should be few rounds
    constexpr int AHEAD = 4;
    const float4* row4 = reinterpret_cast<const float4*>(row);
    const int lo4 = lo >> 2, hi4 = hi >> 2;  // whole vectors; the row's last 1..3 values follow below
    for (int i0 = lo4 + threadIdx.x; i0 < hi4; i0 += AHEAD * blockDim.x) {
      float4 v[AHEAD];
#pragma unroll
      for (int u = 0; u < AHEAD; ++u)
        if (i0 + u * blockDim.x < hi4) v[u] = row4[i0 + u * blockDim.x];
#pragma unroll
      for (int u = 0; u < AHEAD; ++u) {
        const int i = i0 + u * blockDim.x;
        if (i < hi4) {
          if (!isnan(v[u].x)) best = better(best, ArgMax{v[u].x, 4 * i});
          if (!isnan(v[u].y)) best = better(best, ArgMax{v[u].y, 4 * i + 1});
          if (!isnan(v[u].z)) best = better(best, ArgMax{v[u].z, 4 * i + 2});
          if (!isnan(v[u].w)) best = better(best, ArgMax{v[u].w, 4 * i + 3});
        }
      }
    }
    for (int i = (hi4 << 2) + threadIdx.x; i < hi; i += blockDim.x) {
      const float v = row[i];
      if (!isnan(v)) best = better(best, ArgMax{v, i});
    }
  } else {
    for (int i = lo + threadIdx.x; i < hi; i += blockDim.x) {
      const float v = row[i];
      if (!isnan(v)) best = better(best, ArgMax{v, i});
    }
  }
  best = block_argmax(best, scratch);
  if (threadIdx.x == 0) {
    part_v[m * ARGMAX_CHUNKS + c] = best.v;
    part_i[m * ARGMAX_CHUNKS + c] = best.i;
  }
}

__global__ void argmax_final_kernel(const float* __restrict__ part_v, const int* __restrict__ part_i, int* __restrict__ out) {
  JLX_TL(TL_ARGMAX);
  const int m = blockIdx.x, lane = threadIdx.x;
  ArgMax a{part_v[m * ARGMAX_CHUNKS + lane], part_i[m * ARGMAX_CHUNKS + lane]};
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    ArgMax b;
    b.v = __shfl_xor_sync(0xffffffffu, a.v, o);
    b.i = __shfl_xor_sync(0xffffffffu, a.i, o);
    a = better(a, b);
  }
  if (lane == 0) out[m] = a.i < 0 ? 0 : a.i;
}

// part_v: float [M * 32], part_i: int [M * 32] scratch.
JLX_API int jlx_argmax(const float* logits, int M, int V, long long ld, float* part_v, int* part_i, int* out,
                       cudaStream_t stream) {
  JLX_REQUIRE(M >= 0 && V > 0 && ld >= V, "argmax: bad sizes M=%d V=%d", M, V);
  JLX_REQUIRE(part_v && part_i, "argmax: scratch missing");
  JLX_REQUIRE(M <= 65535, "argmax: too many rows");
  if (M == 0) return 0;
  argmax_chunk_kernel<<<dim3(ARGMAX_CHUNKS, M), 256, 0, stream>>>(logits, V, ld, part_v, part_i);
  JLX_LAUNCH_CHECK("argmax_chunk");
  argmax_final_kernel<<<M, 32, 0, stream>>>(part_v, part_i, out);
  JLX_LAUNCH_CHECK("argmax_final");
  return 0;
}

// ---- the variant for callers that cannot allocate: see sampling_noalloc.h for who they are and the rules.
// Layout of the array: ARGMAX_CHUNKS * MAX_ROWS best values (float) followed by as many best indices (int).
static __device__ __align__(256) unsigned char jlx_argmax_noalloc_scratch[JLX_ARGMAX_NOALLOC_MAX_ROWS * ARGMAX_CHUNKS * 8];

// In host code the array's name stands for a host-side shadow, not for device memory: the device address
// has to be asked for, once per device, while that device is current.
static int noalloc_scratch_address(unsigned char** ptr) {
  enum { MAX_DEVICES = 64 };
  static unsigned char* cached[MAX_DEVICES] = {nullptr};
  int dev = -1;
  JLX_CUDA(cudaGetDevice(&dev));
  JLX_REQUIRE(dev >= 0 && dev < MAX_DEVICES, "argmax_noalloc: device ordinal %d is outside 0..%d", dev, MAX_DEVICES - 1);
  if (!cached[dev]) {
    void* p = nullptr;
    JLX_CUDA(cudaGetSymbolAddress(&p, jlx_argmax_noalloc_scratch));
    JLX_REQUIRE(p != nullptr, "argmax_noalloc: the scratch array has no device address");
    cached[dev] = static_cast<unsigned char*>(p);
  }
  *ptr = cached[dev];
  return 0;
}

JLX_API int jlx_argmax_noalloc(const float* logits, int M, int V, long long ld, int* out, cudaStream_t stream) {
  JLX_REQUIRE(M >= 0 && V > 0 && ld >= V, "argmax_noalloc: bad sizes M=%d V=%d", M, V);
  JLX_REQUIRE(M <= JLX_ARGMAX_NOALLOC_MAX_ROWS,
              "argmax_noalloc: %d rows, but the built-in scratch holds %d; use jlx_argmax with your own scratch", M,
              JLX_ARGMAX_NOALLOC_MAX_ROWS);
  JLX_REQUIRE(logits && out, "argmax_noalloc: null input or output");
  if (M == 0) return 0;
  unsigned char* base = nullptr;
  if (noalloc_scratch_address(&base)) return 1;
  float* part_v = reinterpret_cast<float*>(base);
  int* part_i = reinterpret_cast<int*>(base + (size_t)JLX_ARGMAX_NOALLOC_MAX_ROWS * ARGMAX_CHUNKS * sizeof(float));
  // every slot that the second kernel reads (M * ARGMAX_CHUNKS of each half) is written by the first
  argmax_chunk_kernel<<<dim3(ARGMAX_CHUNKS, M), 256, 0, stream>>>(logits, V, ld, part_v, part_i);
  JLX_LAUNCH_CHECK("argmax_chunk");
  argmax_final_kernel<<<M, 32, 0, stream>>>(part_v, part_i, out);
  JLX_LAUNCH_CHECK("argmax_final");
  return 0;
}

JLX_API int jlx_sample_max_top_k() { return SAMPLE_MAX_K; }

// Chunks of a row for sample_top_kernel.  At most SAMPLE_STRAND values per thread (the bound of its candidate list).  8 from
// 16 rows on: 64 rows are then 512 blocks, all resident at once (four an SM).  16 below, where blocks are few: one row of
// 202048, top 64, takes 24 us of which three launches' latency is most.  At least four values per thread: more lists than that
// only lengthen the merging.
static int sample_chunk(int M, int V) {
  const int chunks = M < 16 ? 16 : 8;
  int size = ((V + chunks - 1) / chunks + 3) / 4 * 4;
  if (size < 4 * SAMPLE_THREADS) size = 4 * SAMPLE_THREADS;
  const int most = SAMPLE_THREADS * (SAMPLE_STRAND - 4);  // whole vectors, and one of the last 1..3 values, per thread
  return size < most ? size : most;
}
static long long sample_chunks(int M, int V) { return ((long long)V + sample_chunk(M, V) - 1) / sample_chunk(M, V); }

// Bytes of scratch that jlx_sample needs: the chunks' lists, then the sums of the spans.
JLX_API long long jlx_sample_scratch(int M, int V) {
  if (M <= 0 || V <= 0) return 0;
  return M * (sample_chunks(M, V) * SAMPLE_MAX_K * (long long)sizeof(SampleKey) + SAMPLE_SPANS * (long long)sizeof(float));
}

JLX_API int jlx_sample(const float* logits, int M, int V, long long ld, const float* temperature, const int* top_k,
                       const unsigned long long* streams, const unsigned long long* counters, unsigned long long seed,
                       int* out, void* scratch, cudaStream_t stream) {
  JLX_REQUIRE(M >= 0 && V > 0 && ld >= V, "sample: bad sizes M=%d V=%d", M, V);
  JLX_REQUIRE(!temperature || (streams && counters), "sample: temperature sampling needs streams and counters");
  if (M == 0) return 0;
  JLX_REQUIRE(scratch && ((uintptr_t)scratch & 15) == 0, "sample: scratch missing or not on a 16-byte boundary");
  const long long chunks = sample_chunks(M, V);
  JLX_REQUIRE(chunks <= 65535, "sample: a vocabulary of %d is too large", V);
  SampleKey* lists = (SampleKey*)scratch;
  float* sums = (float*)(lists + (size_t)M * chunks * SAMPLE_MAX_K);
  JLX_CUDA(jlx_launch_pdl(sample_top_kernel, dim3(M, (unsigned)chunks), dim3(SAMPLE_THREADS), 0, stream, logits, V, ld, sample_chunk(M, V),
                          temperature, top_k, lists));
  if (temperature)
    JLX_CUDA(jlx_launch_pdl(sample_spans_kernel, dim3(M, SAMPLE_SPANS / SAMPLE_SPANS_PER_BLOCK), dim3(256), 0, stream, logits, V, ld, (int)chunks,
                            temperature, top_k, lists, sums));
  JLX_CUDA(jlx_launch_pdl(sample_pick_kernel, dim3(M), dim3(SAMPLE_SPANS), 0, stream, logits, V, ld, (int)chunks, temperature, top_k, streams,
                          counters, seed, lists, sums, out));
  JLX_LAUNCH_CHECK("sample");
  return 0;
}
