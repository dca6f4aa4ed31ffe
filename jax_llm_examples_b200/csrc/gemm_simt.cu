// C = A * W^T on the CUDA cores with 32-bit FMA: the matrix product of the true 32-bit path (no
// tensor cores, so no reduced-precision matrix mode can slip in), and of weights that are stored
// in 32-bit while activations are bfloat16.  A: [M, K] row-major, W: [N, K] row-major (the [out, in]
// orientation of the stored Linear weights), C: [M, N].
//
// Grouped form: rows [offsets[e], offsets[e+1]) of A multiply W_e = W + e * w_group_stride
// (the ragged product of llama4/llama4_jax/model.py:975-996).  offsets live on the device, so the
// grid is sized for the worst case and surplus blocks leave at once.
//
// Three kernels; which one runs is decided by sizes alone (gemm_form below):
//
//   gemm_f32_rows   few rows per weight matrix (decode steps, short prompts): every block streams 32 weight rows once for up
//                   to 8 token rows; bound by the weights' bytes.
//   gemm_f32_tile   many rows: tiles of 64 (or 32) x 128 outputs, 8 (4) x 8 per thread; bound by the FMA pipe.
//   gemm_simt       everything that is not float32 throughout or not in whole 16-byte pieces.
//
// The order in which an output's K products are added does not depend on the number of rows, so that a position's result does
// not depend on how its prompt was cut into steps.  The two float32 kernels share one order, which follows from K alone: four
// parts of whole 32s; a part has a strand of its even and one of its odd K, each one by one; the strands are added, then the
// parts in order.  gemm_simt adds the products one by one; a product's types, leading dimensions and addresses send it there.

#include "common.cuh"

#define BM 64
#define BN 64
#define BK 16
#define LDS 68  // padded row of the shared tiles (floats); 16-byte aligned for float4 reads

template <typename TA, typename TW, typename TC>
__global__ void __launch_bounds__(256)
gemm_simt_kernel(const TA* __restrict__ A, const TW* __restrict__ W, TC* __restrict__ C, int M, int N, int K,
                 long long lda, long long ldw, long long ldc, const int* __restrict__ offsets, int E,
                 long long w_group_stride) {
  JLX_TL(TL_GEMM_SIMT);
  __shared__ __align__(16) float As[BK][LDS];
  __shared__ __align__(16) float Ws[BK][LDS];

  int m0, m_end;
  const TW* Wg = W;
  if (offsets) {
    // find this block's (group, row tile)
    int t = blockIdx.y, e = 0, found = 0;
    for (; e < E; ++e) {
      const int lo = offsets[e], hi = offsets[e + 1];
      const int tiles = (hi - lo + BM - 1) / BM;
      if (t < tiles) {
        m0 = lo + t * BM;
        m_end = hi;
        found = 1;
        break;
      }
      t -= tiles;
    }
    if (!found) return;
    Wg = W + (size_t)e * w_group_stride;
  } else {
    m0 = blockIdx.y * BM;
    m_end = M;
    if (m0 >= M) return;
  }
  const int n0 = blockIdx.x * BN;
  const int tid = threadIdx.x;
  const int tx = tid & 15, ty = tid >> 4;
  const int lr = tid >> 2, lk = (tid & 3) * 4;  // loader: row 0..63, k offset 0,4,8,12

  float acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;

  for (int k0 = 0; k0 < K; k0 += BK) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int k = k0 + lk + j;
      const int am = m0 + lr, wn = n0 + lr;
      As[lk + j][lr] = (am < m_end && k < K) ? to_f32<TA>(A[(size_t)am * lda + k]) : 0.f;
      Ws[lk + j][lr] = (wn < N && k < K) ? to_f32<TW>(Wg[(size_t)wn * ldw + k]) : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < BK; ++k) {
      const float4 a = *reinterpret_cast<const float4*>(&As[k][ty * 4]);
      const float4 b = *reinterpret_cast<const float4*>(&Ws[k][tx * 4]);
      const float av[4] = {a.x, a.y, a.z, a.w}, bv[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(av[i], bv[j], acc[i][j]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int m = m0 + ty * 4 + i;
    if (m >= m_end) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int n = n0 + tx * 4 + j;
      if (n < N) C[(size_t)m * ldc + n] = from_f32<TC>(acc[i][j]);
    }
  }
}

// ------------------------------------------------------------------------------------------------ float32 throughout
// Two 32-bit products per instruction; each half is the IEEE fused multiply-add.
__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
  unsigned long long d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ unsigned long long pair_of(float x, float y) {
  return (unsigned long long)__float_as_uint(x) | ((unsigned long long)__float_as_uint(y) << 32);
}
__device__ __forceinline__ float low_of(unsigned long long p) { return __uint_as_float((unsigned)p); }
__device__ __forceinline__ float high_of(unsigned long long p) { return __uint_as_float((unsigned)(p >> 32)); }

// The group and the rows [m0, m_end) of row tile t, tiles of `rows` rows, groups one after the other; false: no such tile.
// Each lane looks at one group of every 32, so that the offsets cost one round trip and not one per group.
__device__ __forceinline__ bool find_row_tile(const int* __restrict__ offsets, int E, int t, int rows, int& group, int& m0, int& m_end) {
  const int lane = threadIdx.x & 31;
  for (int e0 = 0; e0 < E; e0 += 32) {
    const int e = e0 + lane;
    const int lo = e < E ? offsets[e] : 0, hi = e < E ? offsets[e + 1] : 0;
    const int tiles = (hi - lo + rows - 1) / rows;
    int upto = tiles;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int x = __shfl_up_sync(0xffffffffu, upto, o);
      if (lane >= o) upto += x;
    }
    const unsigned past = __ballot_sync(0xffffffffu, upto > t);
    if (past) {
      const int src = __ffs(past) - 1;
      group = e0 + src;
      m0 = __shfl_sync(0xffffffffu, lo + (t - (upto - tiles)) * rows, src);
      m_end = __shfl_sync(0xffffffffu, hi, src);
      return true;
    }
    t -= __shfl_sync(0xffffffffu, upto, 31);
  }
  return false;
}

#define GEMM_PARTS 4
__host__ __device__ __forceinline__ int gemm_part(int K) { return ((K + GEMM_PARTS - 1) / GEMM_PARTS + 31) / 32 * 32; }

__device__ __forceinline__ void copy16_or_zero(float* dst, const float* src, bool there) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src), "r"(there ? 16 : 0) : "memory");
}

// 8 RM x 128 outputs per block of 128 threads: a warp 4 RM x 64, a thread RM rows by 8 columns.  A packed FMA takes two
// neighbouring K of a row of A and of a row of W as they lie in memory (the two strands), nothing is transposed, and the K
// slices come by 16-byte asynchronous copies into a ring of four.  A thread's rows are every fourth, its columns every
// eighth, and a row of a slice is 80 bytes: the lanes that read together read different banks.  Four K of RM = 8 are sixteen
// 16-byte reads for 128 packed FMAs.  The parts before a block's last are added up in a place beside the ring.
// Where the tiles are too few for the GPU, a cluster of two or four blocks shares the parts and adds them through
// distributed shared memory.
// Bound by the FMA pipe, whose rate with such operands is about 60 TFLOP/s (32 independent accumulators in registers,
// nothing else), and by the reads beside it: 1024 x 8192 x 2048 takes
// 817 us (42 TFLOP/s; the kernel with 64 x 64 tiles and scalar loads, above, 1360), 1024 x 3072 x 2048 338 us (600).
#define TN 128
#define TK 16
#define TILE_LD 20  // floats per row of a slice
#define TILE_STAGES 4
#define SUM_LD (TN + 4)
template <int RM>
__global__ void __launch_bounds__(128, 2)
gemm_f32_tile_kernel(const float* __restrict__ A, const float* __restrict__ W, float* __restrict__ C, int M, int N, int K, long long lda,
                     long long ldw, long long ldc, const int* __restrict__ offsets, int E, long long w_group_stride) {
  JLX_TL(TL_GEMM_SIMT);
  constexpr int TM = 8 * RM, STAGE = (TM + TN) * TILE_LD;
  extern __shared__ __align__(16) float ring[];  // [TILE_STAGES][TM rows of A, then TN rows of W][TILE_LD]; then the sums' place
  float* before = ring + TILE_STAGES * STAGE;    // [TM][SUM_LD]: the parts before the block's last
  int m0 = blockIdx.x * TM, m_end = M, group = 0;
  if (offsets && !find_row_tile(offsets, E, blockIdx.x, TM, group, m0, m_end)) return;  // all blocks of a cluster alike
  const float* Wg = W + (size_t)group * w_group_stride;
  const int n0 = blockIdx.y * TN;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int mt = (warp >> 1) * (4 * RM) + (lane >> 3), nt = (warp & 1) * 64 + (lane & 7);  // rows mt + 4 i, columns nt + 8 j
  const int shares = gridDim.z, own = GEMM_PARTS / shares, part = gemm_part(K);
  const int k_first = min(K, (int)blockIdx.z * own * part), k_end = min(K, ((int)blockIdx.z + 1) * own * part);
  // loader: four threads per row, 32 rows at a time; rows past the end read a row that is there and are not stored
  const int lr = tid >> 2, lk = (tid & 3) * 4;
  const float* ap[TM / 32];
  const float* wp[TN / 32];
#pragma unroll
  for (int i = 0; i < TM / 32; ++i) ap[i] = A + (size_t)min(m0 + lr + 32 * i, m_end - 1) * lda + lk;
#pragma unroll
  for (int i = 0; i < TN / 32; ++i) wp[i] = Wg + (size_t)min(n0 + lr + 32 * i, N - 1) * ldw + lk;
  auto fetch = [&](int k0, int stage) {  // always a group of copies, maybe an empty one
    if (k0 < k_end) {
      const bool there = k0 + lk < k_end;  // K and the parts of it are multiples of 4
      const int at = there ? k0 : -lk;     // (an address that exists, of which nothing is read)
      float* dst = ring + stage * STAGE + lr * TILE_LD + lk;
#pragma unroll
      for (int i = 0; i < TM / 32; ++i) copy16_or_zero(dst + 32 * i * TILE_LD, ap[i] + at, there);
#pragma unroll
      for (int i = 0; i < TN / 32; ++i) copy16_or_zero(dst + (TM + 32 * i) * TILE_LD, wp[i] + at, there);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  unsigned long long acc[RM][8];
#pragma unroll
  for (int i = 0; i < RM; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[i][j] = 0ull;
#pragma unroll
  for (int g = 0; g < TILE_STAGES - 1; ++g) fetch(k_first + g * TK, g);
  int stage = 0, part_end = k_first + part;
  bool first = true;
  for (int k0 = k_first; k0 < k_end; k0 += TK) {
    if (k0 == part_end) {  // (a part is whole slices) every thread keeps its own outputs' sums
#pragma unroll
      for (int i = 0; i < RM; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          float* at = before + (mt + 4 * i) * SUM_LD + nt + 8 * j;
          const float s = low_of(acc[i][j]) + high_of(acc[i][j]);
          *at = first || (shares > 1 && blockIdx.z > 0) ? s : *at + s;  // (two blocks: the second has one part here)
          acc[i][j] = 0ull;
        }
      first = false;
      part_end += part;
    }
    asm volatile("cp.async.wait_group %0;" ::"n"(TILE_STAGES - 2) : "memory");
    __syncthreads();  // this slice is there for everyone, and everyone is past the slice whose place is filled next
    fetch(k0 + (TILE_STAGES - 1) * TK, (stage + TILE_STAGES - 1) % TILE_STAGES);
    const float* as = ring + stage * STAGE + mt * TILE_LD;
    const float* ws = ring + stage * STAGE + (TM + nt) * TILE_LD;
#pragma unroll
    for (int k = 0; k < TK; k += 4) {
      ulonglong2 w[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) w[j] = *reinterpret_cast<const ulonglong2*>(ws + 8 * j * TILE_LD + k);
#pragma unroll
      for (int i = 0; i < RM; ++i) {
        const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(as + 4 * i * TILE_LD + k);
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[i][j] = fma2(a.x, w[j].x, acc[i][j]);
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[i][j] = fma2(a.y, w[j].y, acc[i][j]);
      }
    }
    stage = (stage + 1) % TILE_STAGES;
  }
  __syncthreads();  // the ring's last slice is read: its place serves the sums (no copies are in flight any more)
  float* sums = ring;  // [TM][SUM_LD]: the first block of a cluster, or the only one: all its parts; the others: the last part
  const bool second = shares == 2 && blockIdx.z == 1;
#pragma unroll
  for (int i = 0; i < RM; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int at = (mt + 4 * i) * SUM_LD + nt + 8 * j;
      const float s = low_of(acc[i][j]) + high_of(acc[i][j]);
      sums[at] = first || second ? s : before[at] + s;
      if (second && first) before[at] = 0.f;  // K ends inside the block's first part, whose sums are in `sums`
    }
  if (shares == 1) __syncthreads();
  else asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
  const bool vec = (ldc & 3) == 0 && ((uintptr_t)C & 15) == 0;
  for (int idx = blockIdx.z * 128 + tid; idx < TM * (TN / 4); idx += shares * 128) {
    const int r = idx / (TN / 4), c = idx % (TN / 4) * 4, m = m0 + r, n = n0 + c;
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (shares == 1) v = *reinterpret_cast<float4*>(sums + r * SUM_LD + c);
    auto add = [&](const float* mine, int z) {
      uint32_t there;
      float4 x;
      asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(there) : "r"((uint32_t)__cvta_generic_to_shared(mine)), "r"(z));
      asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(x.x), "=f"(x.y), "=f"(x.z), "=f"(x.w) : "r"(there) : "memory");
      v = make_float4(v.x + x.x, v.y + x.y, v.z + x.z, v.w + x.w);
    };
    for (int z = 0; shares > 1 && z < shares; ++z) {
      if (shares == 2 && z == 1) add(before + r * SUM_LD + c, z);
      add(sums + r * SUM_LD + c, z);
    }
    if (m >= m_end) continue;
    float* dst = C + (size_t)m * ldc + n;
    if (vec && n + 3 < N) {
      *reinterpret_cast<float4*>(dst) = v;
    } else {
      const float e[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (n + j < N) dst[j] = e[j];
    }
  }
  if (shares > 1)  // the others may still read here
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

template <int RM>
static cudaError_t launch_tile(const float* a, const float* w, float* c, int M, int N, int K, long long lda, long long ldw, long long ldc,
                               const int* offsets, int E, long long wgs, int shares, cudaStream_t stream) {
  const int smem = (int)sizeof(float) * (TILE_STAGES * (8 * RM + TN) * TILE_LD + 8 * RM * SUM_LD);
  const cudaError_t e = cudaFuncSetAttribute(gemm_f32_tile_kernel<RM>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)((M + 8 * RM - 1) / (8 * RM) + (offsets ? E : 0)), (N + TN - 1) / TN, shares);
  cfg.blockDim = dim3(128);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 1;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = shares;
  cfg.attrs = attr;
  cfg.numAttrs = shares > 1 ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, gemm_f32_tile_kernel<RM>, a, w, c, M, N, K, lda, ldw, ldc, offsets, E, wgs);
}

// MT token rows by 32 weight rows per block of four warps, one for each part of K; a lane has a weight row.  Every warp
// brings its own slices of 32 K into a ring of its own (a row of a slice is 144 bytes: eight lanes read eight different
// 16-byte columns of banks), so the warps meet only once, when the parts are added.  Blocks that share weight rows follow
// one another: more than MT token rows read them from L2 again.
// Bound by the weights' bytes, and with few columns by how much a block's four rings keep in flight: one
// row by 8192 x 2048 takes 25 us (67 MB, 10 us at the copy rate), 32768 x 2048 66 us (41); the tiles of the general kernel
// took 156 and 365.
#define RN 32
#define ROWS_K 32
#define ROWS_LD 36
#define ROWS_STAGES 4
template <int MT>
__global__ void __launch_bounds__(128)
gemm_f32_rows_kernel(const float* __restrict__ A, const float* __restrict__ W, float* __restrict__ C, int M, int N, int K, long long lda,
                     long long ldw, long long ldc, const int* __restrict__ offsets, int E, long long w_group_stride) {
  JLX_TL(TL_GEMM_SIMT);
  constexpr int STAGE = (RN + MT) * ROWS_LD;
  extern __shared__ __align__(16) float rings[];  // [warp][stage][weight rows, then token rows][ROWS_LD]
  __shared__ float sums[GEMM_PARTS][MT][RN];
  int m0 = blockIdx.x * MT, m_end = M, group = 0;
  if (offsets && !find_row_tile(offsets, E, blockIdx.x, MT, group, m0, m_end)) return;
  const float* Wg = W + (size_t)group * w_group_stride;
  const int n0 = blockIdx.y * RN;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, part = gemm_part(K);
  const int k_first = min(K, warp * part), k_end = min(K, k_first + part);
  float* ring = rings + warp * ROWS_STAGES * STAGE;
  // loader: eight lanes per row, four rows at a time
  const int lr = lane >> 3, lk = (lane & 7) * 4;
  auto fetch = [&](int k0, int stage) {  // always a group of copies, maybe an empty one
    if (k0 < k_end) {
      const bool there = k0 + lk < k_end;
      const int at = there ? k0 + lk : 0;
      float* dst = ring + stage * STAGE + lr * ROWS_LD + lk;
#pragma unroll
      for (int i = 0; i < RN / 4; ++i) copy16_or_zero(dst + 4 * i * ROWS_LD, Wg + (size_t)min(n0 + lr + 4 * i, N - 1) * ldw + at, there);
#pragma unroll
      for (int i = 0; i < (MT + 3) / 4; ++i)
        if (lr + 4 * i < MT) copy16_or_zero(dst + (RN + 4 * i) * ROWS_LD, A + (size_t)min(m0 + lr + 4 * i, m_end - 1) * lda + at, there);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  unsigned long long acc[MT];
#pragma unroll
  for (int i = 0; i < MT; ++i) acc[i] = 0ull;
#pragma unroll
  for (int g = 0; g < ROWS_STAGES - 1; ++g) fetch(k_first + g * ROWS_K, g);
  int stage = 0;
  for (int k0 = k_first; k0 < k_end; k0 += ROWS_K) {
    asm volatile("cp.async.wait_group %0;" ::"n"(ROWS_STAGES - 2) : "memory");
    __syncwarp();  // this slice is there for the warp, and the warp is past the slice whose place is filled next
    fetch(k0 + (ROWS_STAGES - 1) * ROWS_K, (stage + ROWS_STAGES - 1) % ROWS_STAGES);
    const float* ws = ring + stage * STAGE + lane * ROWS_LD;
    const float* as = ring + stage * STAGE + RN * ROWS_LD;
#pragma unroll
    for (int k = 0; k < ROWS_K; k += 4) {
      const ulonglong2 w = *reinterpret_cast<const ulonglong2*>(ws + k);
#pragma unroll
      for (int i = 0; i < MT; ++i) {
        const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(as + i * ROWS_LD + k);
        acc[i] = fma2(a.y, w.y, fma2(a.x, w.x, acc[i]));
      }
    }
    stage = (stage + 1) % ROWS_STAGES;
  }
#pragma unroll
  for (int i = 0; i < MT; ++i) sums[warp][i][lane] = low_of(acc[i]) + high_of(acc[i]);
  __syncthreads();
  for (int idx = threadIdx.x; idx < MT * RN; idx += 128) {
    const int i = idx / RN, n = idx % RN;
    if (m0 + i >= m_end || n0 + n >= N) continue;
    float s = sums[0][i][n];
#pragma unroll
    for (int p = 1; p < GEMM_PARTS; ++p) s += sums[p][i][n];
    C[(size_t)(m0 + i) * ldc + n0 + n] = s;
  }
}

template <int MT>
static cudaError_t launch_rows(const float* a, const float* w, float* c, int M, int N, int K, long long lda, long long ldw, long long ldc,
                               const int* offsets, int E, long long wgs, cudaStream_t stream) {
  const int smem = (int)sizeof(float) * GEMM_PARTS * ROWS_STAGES * (RN + MT) * ROWS_LD;
  const cudaError_t e = cudaFuncSetAttribute(gemm_f32_rows_kernel<MT>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return e;
  const dim3 grid((unsigned)((M + MT - 1) / MT + (offsets ? (E < M ? E : M) : 0)), (N + RN - 1) / RN);
  gemm_f32_rows_kernel<MT><<<grid, 128, smem, stream>>>(a, w, c, M, N, K, lda, ldw, ldc, offsets, E, wgs);
  return cudaGetLastError();
}

template <typename TA, typename TW, typename TC>
static int launch(const void* A, const void* W, void* C, int M, int N, int K, long long lda, long long ldw,
                  long long ldc, const int* offsets, int E, long long wgs, cudaStream_t stream) {
  const int row_tiles = (M + BM - 1) / BM + (offsets ? E : 0);
  JLX_REQUIRE(row_tiles <= 65535, "gemm_simt: too many row tiles (%d)", row_tiles);
  dim3 grid((N + BN - 1) / BN, row_tiles);
  gemm_simt_kernel<TA, TW, TC><<<grid, 256, 0, stream>>>((const TA*)A, (const TW*)W, (TC*)C, M, N, K, lda, ldw, ldc,
                                                        offsets, E, wgs);
  JLX_LAUNCH_CHECK("gemm_simt");
  return 0;
}

enum { GEMM_FORM_RULE = 0, GEMM_FORM_GENERAL = 1, GEMM_FORM_TILE = 2, GEMM_FORM_ROWS = 3 };

// Which kernel, by estimates of the time in microseconds on this GPU (148 multiprocessors), fitted to measurements at N x K
// from 2048 x 2048 to 32768 x 2048 with 1 to 1024 rows, dense and in 8 groups:
//   rows: 0.5 us per million weights for their bytes and 0.35 to 0.65 for every tile of 1 to 8 rows.
//   tile: a multiprocessor takes 53 ns per K and tile of 64 rows, 31 ns of 32 rows; a lone block 64 and 38; cutting K over
//         a cluster costs 3 us.
// (32768 x 2048, 8 rows: rows 80, 32-row tiles 141; 8192 x 2048, 16 rows: rows 41, 32-row tiles cut in four 45; 32 rows: 78 and
// 45; 64 rows: rows 135, 64-row tiles cut in four 72; 1024 rows: rows 2034, 64-row tiles 817; 64 rows in 8 groups: rows 180,
// 32-row tiles 238.)
struct GemmPlan { int form, rm, shares, mt; };
static GemmPlan gemm_plan(int M, int N, int K, int groups) {
  const int per = (M + groups - 1) / groups;  // rows that a weight matrix typically multiplies
  const int mt = per <= 1 ? 1 : (per <= 2 ? 2 : (per <= 4 ? 4 : 8));
  double missed = 1.0;  // the share of groups that M rows spread at random leave without one
  for (int i = 0; groups > 1 && i < M && missed > 0.01; ++i) missed *= 1.0 - 1.0 / groups;
  const double used = groups > 1 ? groups * (1.0 - missed) : 1.0, million = (double)K * N * 1e-6;
  auto row_tiles = [&](int size) {  // a group's last tile is half full
    const double t = (double)M / size + (groups > 1 && size > 1 ? 0.5 * used : 0.0);
    return groups > 1 ? (t > used ? t : used) : (double)((M + size - 1) / size);
  };
  GemmPlan best = {GEMM_FORM_ROWS, 0, 1, mt};
  double least = 5.0 + million * (0.5 * used + (mt == 1 ? 0.35 : (mt == 2 ? 0.4 : (mt == 4 ? 0.6 : 0.65))) * row_tiles(mt));
  for (int rm = 4; rm <= 8; rm += 4)
    for (int shares = 1; shares <= GEMM_PARTS && (shares == 1 || K / shares >= 256); shares *= 2) {
      const double blocks = row_tiles(8 * rm) * ((N + TN - 1) / TN) * shares;
      const double rounds = blocks <= 148 ? 1.0 : (double)(long long)(blocks / 148 + 0.999);
      const double per_k = rounds <= 1.0 ? (rm == 8 ? 0.064 : 0.038) : rounds * (rm == 8 ? 0.053 : 0.031);
      const double t = per_k * K / shares + (shares > 1 ? 3.0 : 0.0);
      if (t < least) {
        least = t;
        best = {GEMM_FORM_TILE, rm, shares, mt};
      }
    }
  return best;
}

// M is the row count (dense) or an upper bound of offsets[E] (grouped).  form: GEMM_FORM_RULE, or the kernel to run (a test's).
JLX_API int jlx_gemm_simt(const void* A, int a_dtype, const void* W, int w_dtype, void* C, int c_dtype, int M, int N,
                          int K, long long lda, long long ldw, long long ldc, const int* offsets, int E,
                          long long w_group_stride, int form, cudaStream_t stream) {
  JLX_REQUIRE(M >= 0 && N > 0 && K > 0, "gemm_simt: bad sizes M=%d N=%d K=%d", M, N, K);
  JLX_REQUIRE(lda >= K && ldw >= K && ldc >= N, "gemm_simt: a leading dimension is smaller than its row");
  JLX_REQUIRE(!offsets || E > 0, "gemm_simt: grouped product needs a group count");
  if (M == 0) return 0;
  const int code = a_dtype * 4 + w_dtype * 2 + c_dtype;
  const bool pieces = code == 0 && K % 4 == 0 && lda % 4 == 0 && ldw % 4 == 0 && w_group_stride % 4 == 0 &&
                      (((uintptr_t)A | (uintptr_t)W) & 15) == 0;
  JLX_REQUIRE(form == GEMM_FORM_RULE || form == GEMM_FORM_GENERAL || pieces, "gemm_simt: this form takes float32 in whole 16-byte pieces");
  GemmPlan plan = pieces ? gemm_plan(M, N, K, offsets ? E : 1) : GemmPlan{GEMM_FORM_GENERAL, 0, 1, 1};
  if (form == GEMM_FORM_TILE && plan.form != form) plan = {form, 4, K >= 512 ? 2 : 1, 8};
  if (form == GEMM_FORM_RULE) form = plan.form;
  const float *a = (const float*)A, *w = (const float*)W;
  const long long groups = offsets ? E : 0;
  if (form == GEMM_FORM_TILE && (N + TN - 1) / TN <= 65535) {
#define TILE(RM) JLX_CUDA(launch_tile<RM>(a, w, (float*)C, M, N, K, lda, ldw, ldc, offsets, E, w_group_stride, plan.shares, stream))
    if (plan.rm == 8) TILE(8);
    else TILE(4);
#undef TILE
    JLX_LAUNCH_CHECK("gemm_f32_tile");
    return 0;
  }
  if (form == GEMM_FORM_ROWS && (N + RN - 1) / RN <= 65535) {
    JLX_CUDA(plan.mt == 1 ? launch_rows<1>(a, w, (float*)C, M, N, K, lda, ldw, ldc, offsets, E, w_group_stride, stream)
             : plan.mt == 2 ? launch_rows<2>(a, w, (float*)C, M, N, K, lda, ldw, ldc, offsets, E, w_group_stride, stream)
             : plan.mt == 4 ? launch_rows<4>(a, w, (float*)C, M, N, K, lda, ldw, ldc, offsets, E, w_group_stride, stream)
                            : launch_rows<8>(a, w, (float*)C, M, N, K, lda, ldw, ldc, offsets, E, w_group_stride, stream));
    JLX_LAUNCH_CHECK("gemm_f32_rows");
    return 0;
  }
#define GO(TA, TW, TC) return launch<TA, TW, TC>(A, W, C, M, N, K, lda, ldw, ldc, offsets, E, w_group_stride, stream)
  switch (code) {
    case 0: GO(float, float, float);
    case 1: GO(float, float, bf16);
    case 2: GO(float, bf16, float);
    case 3: GO(float, bf16, bf16);
    case 4: GO(bf16, float, float);
    case 5: GO(bf16, float, bf16);
    case 6: GO(bf16, bf16, float);
    case 7: GO(bf16, bf16, bf16);
  }
#undef GO
  JLX_REQUIRE(false, "gemm_simt: unknown element type codes %d %d %d", a_dtype, w_dtype, c_dtype);
}
