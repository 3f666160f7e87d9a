// General tiled GEMM on CUDA cores with fp32 accumulation: fp32 products that are too small or too short for
// gemm_f32_umma.cu, or off the 16-byte grid, and bf16 shapes the tcgen05 path does not take (tiny K, unaligned strides).  y = epilogue(x @ W^T).
//
// Bound: FFMA issue (74 TFLOP/s), and before that the number of CTAs: the prefill linears of a 512-wide fp32 model are
// 256 x 512 x 6144.  64 x 64 tiles of 128 threads (8 x 4 outputs each: three 16-byte shared-memory reads per 32 FMAs)
// with K split over a thread-block cluster of up to 8 CTAs until there are about two per SM (the partial tiles meet in
// distributed shared memory, summed in rank order).  (128 x 128 tiles of 8 x 8 outputs where those alone fill the chip
// are 2 to 5 % ahead only for the largest products, 4000 x 8192 x 4096 6.01 against 6.30 ms, and fall far behind on
// short K, where the outputs leave in rows of 8: 8192 x 1024 x 24, the taps of an STU layer, 47 against 20 us.)
// Operand tiles pass through registers into a double-buffered, k-major shared-memory tile.  256 x 512 x 6144:
// 531 us with 64 x 64 tiles of 4 x 4 outputs, no split and no overlap.
#include <cooperative_groups.h>

#include "common.cuh"
#include "epilogue.cuh"

int device_sm_count();   // gemm_tc.cu

namespace cg = cooperative_groups;

namespace {

constexpr int BM = 64, BK = 16;    // tile (BN 64 or 32)
constexpr int TM = 8, TN = 4;      // outputs of a thread

// Four consecutive k of one row as fp32; vec: 16-byte (fp32) / 8-byte (bf16) aligned and inside the row.
__device__ __forceinline__ void load4(const float* p, float (&v)[4]) {
  const float4 t = *reinterpret_cast<const float4*>(p);
  v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
}
__device__ __forceinline__ void load4(const bf16* p, float (&v)[4]) {
  const uint2 t = *reinterpret_cast<const uint2*>(p);
  v[0] = __uint_as_float(t.x << 16);
  v[1] = __uint_as_float(t.x & 0xffff0000u);
  v[2] = __uint_as_float(t.y << 16);
  v[3] = __uint_as_float(t.y & 0xffff0000u);
}

// KS > 1: cluster of KS CTAs along z.
template <typename T, int EPI, int KS, int BN>
__global__ void __launch_bounds__(BM / TM * (BN / TN))
    gemm_simt_kernel(const T* __restrict__ A, long long lda, const T* __restrict__ B, long long ldb, long long skb,
                     const T* __restrict__ B2, int M, int N, int K, int causal, int vec_a, int vec_b, EpiArgs<T> ep) {
  constexpr bool DUAL = (EPI == EPI_GELU_MUL);
  constexpr int NB = DUAL ? 2 : 1;
  constexpr int TX = BN / TN, THREADS = BM / TM * TX;                     // threads across the columns, in all
  constexpr int QA = BM * BK / 4 / THREADS, QB = BN * BK / 4 / THREADS;   // quads of k per thread and tile
  static_assert(QA >= 1 && QB >= 1, "thread layout");
  constexpr int PA = BM + 4, PB = BN + 4;
  constexpr int TILE = BK * (PA + NB * PB);
  constexpr int PART = KS > 1 ? BM * BN * NB : 0;
  __shared__ __align__(16) float sm[2 * TILE > PART ? 2 * TILE : PART];
  const int tid = threadIdx.x, tx = tid % TX, ty = tid / TX;
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  const int k_end = causal ? min(K, n0 + BN) : K;   // a lower-triangular B has nothing beyond the tile's last column

  const int nkb = (k_end + BK - 1) / BK, per = (nkb + KS - 1) / KS;
  const int kb0 = KS > 1 ? (int)blockIdx.z * per : 0, kb1 = KS > 1 ? min(nkb, kb0 + per) : nkb;

  float ra[QA][4], rb[NB][QB][4];
  auto fetch = [&](int kb) {
    const int k0 = kb * BK;
#pragma unroll
    for (int i = 0; i < QA; i++) {
      const int e = tid + i * THREADS, r = e >> 2, k = k0 + (e & 3) * 4, m = m0 + r;
      const T* p = A + (size_t)m * lda + k;
      if (m < M && vec_a && k + 4 <= K) {
        load4(p, ra[i]);
      } else {
#pragma unroll
        for (int j = 0; j < 4; j++) ra[i][j] = (m < M && k + j < K) ? Elem<T>::to_f(p[j]) : 0.f;
      }
    }
#pragma unroll
    for (int b = 0; b < NB; b++)
#pragma unroll
      for (int i = 0; i < QB; i++) {
        const int e = tid + i * THREADS, r = e >> 2, k = k0 + (e & 3) * 4, n = n0 + r;
        const T* p = (b ? B2 : B) + (size_t)n * ldb + (size_t)k * skb;
        if (n < N && vec_b && k + 4 <= K) {
          load4(p, rb[b][i]);
        } else {
#pragma unroll
          for (int j = 0; j < 4; j++) rb[b][i][j] = (n < N && k + j < K) ? Elem<T>::to_f(p[(size_t)j * skb]) : 0.f;
        }
      }
  };
  auto stage = [&](int buf) {
    float* a = sm + buf * TILE;
#pragma unroll
    for (int i = 0; i < QA; i++) {
      const int e = tid + i * THREADS, r = e >> 2, k = (e & 3) * 4;
#pragma unroll
      for (int j = 0; j < 4; j++) a[(k + j) * PA + r] = ra[i][j];
    }
#pragma unroll
    for (int b = 0; b < NB; b++) {
      float* bs = a + BK * PA + b * BK * PB;
#pragma unroll
      for (int i = 0; i < QB; i++) {
        const int e = tid + i * THREADS, r = e >> 2, k = (e & 3) * 4;
#pragma unroll
        for (int j = 0; j < 4; j++) bs[(k + j) * PB + r] = rb[b][i][j];
      }
    }
  };

  float acc[NB][TM][TN];
#pragma unroll
  for (int b = 0; b < NB; b++)
#pragma unroll
    for (int i = 0; i < TM; i++)
#pragma unroll
      for (int j = 0; j < TN; j++) acc[b][i][j] = 0.f;

  if (kb0 < kb1) {
    fetch(kb0);
    stage(0);
  }
  __syncthreads();
  for (int kb = kb0; kb < kb1; kb++) {
    const int buf = (kb - kb0) & 1;
    if (kb + 1 < kb1) fetch(kb + 1);   // in flight during the products below
    const float* a = sm + buf * TILE + ty * TM;
    const float* bs = sm + buf * TILE + BK * PA + tx * TN;
#pragma unroll
    for (int kk = 0; kk < BK; kk++) {
      float av[TM], bv[NB][TN];
#pragma unroll
      for (int i = 0; i < TM; i += 4) *reinterpret_cast<float4*>(av + i) = *reinterpret_cast<const float4*>(a + kk * PA + i);
#pragma unroll
      for (int b = 0; b < NB; b++)
#pragma unroll
        for (int j = 0; j < TN; j += 4)
          *reinterpret_cast<float4*>(bv[b] + j) = *reinterpret_cast<const float4*>(bs + b * BK * PB + kk * PB + j);
#pragma unroll
      for (int b = 0; b < NB; b++)
#pragma unroll
        for (int i = 0; i < TM; i++)
#pragma unroll
          for (int j = 0; j < TN; j++) acc[b][i][j] = fmaf(av[i], bv[b][j], acc[b][i][j]);
    }
    if (kb + 1 < kb1) stage(buf ^ 1);   // the other buffer was last read before the barrier of the step before
    __syncthreads();
  }

  if constexpr (KS == 1) {
#pragma unroll
    for (int i = 0; i < TM; i++)
#pragma unroll
      for (int j = 0; j < TN; j++) {
        const int m = m0 + ty * TM + i, n = n0 + tx * TN + j;
        if (m < M && n < N) epilogue_store<T, EPI>(ep, m, n, acc[0][i][j], DUAL ? acc[NB - 1][i][j] : 0.f);
      }
  } else {
    cg::cluster_group cluster = cg::this_cluster();
#pragma unroll
    for (int b = 0; b < NB; b++)
#pragma unroll
      for (int i = 0; i < TM; i++)
#pragma unroll
        for (int j = 0; j < TN; j += 4)
          *reinterpret_cast<float4*>(sm + (b * BM + ty * TM + i) * BN + tx * TN + j) =
              make_float4(acc[b][i][j], acc[b][i][j + 1], acc[b][i][j + 2], acc[b][i][j + 3]);
    cluster.sync();   // every partial tile is complete
    const int rank = (int)cluster.block_rank();
    const float* part[KS];
#pragma unroll
    for (int r = 0; r < KS; r++) part[r] = cluster.map_shared_rank(sm, r);
    for (int e = tid; e < BM / KS * BN; e += THREADS) {   // every CTA finishes its share of the rows
      const int row = rank + (e / BN) * KS, col = e % BN, m = m0 + row, n = n0 + col;
      float s = 0.f, s2 = 0.f;
#pragma unroll
      for (int r = 0; r < KS; r++) {
        s += part[r][row * BN + col];
        if (DUAL) s2 += part[r][(BM + row) * BN + col];
      }
      if (m < M && n < N) epilogue_store<T, EPI>(ep, m, n, s, s2);
    }
    cluster.sync();   // the other CTAs' tiles stay alive until read
  }
}

struct Operands {
  const void *A, *B, *B2;
  long long lda, ldb, skb;
  int M, N, K, causal, vec_a, vec_b;
};

template <typename T, int EPI, int KS, int BN>
int launch_tile(const Operands& o, const EpiArgs<T>& ep, cudaStream_t st) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((o.N + BN - 1) / BN, (o.M + BM - 1) / BM, KS);
  cfg.blockDim = dim3(BM / TM * (BN / TN));
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = 1;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = KS;
  cfg.attrs = at;
  cfg.numAttrs = KS > 1 ? 1 : 0;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, gemm_simt_kernel<T, EPI, KS, BN>, (const T*)o.A, o.lda,
                                           (const T*)o.B, o.ldb, o.skb, (const T*)o.B2, o.M, o.N, o.K, o.causal, o.vec_a,
                                           o.vec_b, ep);
  if (e != cudaSuccess) return (int)e;
  STU_CHECK_LAUNCH();
  return STU_OK;
}

template <typename T, int EPI, int BN>
int launch_simt(const Operands& o, const EpiArgs<T>& ep, cudaStream_t st) {
  const long long sms = device_sm_count(), tiles = (long long)((o.M + BM - 1) / BM) * ((o.N + BN - 1) / BN);
  // split K while there are fewer than two CTAs of 64 columns (or their like in threads) per SM and every CTA keeps 64 of K
  int ks = 1;
  while (ks < 8 && tiles * ks * BN < 2 * sms * 64 && o.K / (2 * ks) >= 64) ks *= 2;
  switch (ks) {
    case 1: return launch_tile<T, EPI, 1, BN>(o, ep, st);
    case 2: return launch_tile<T, EPI, 2, BN>(o, ep, st);
    case 4: return launch_tile<T, EPI, 4, BN>(o, ep, st);
    default: return launch_tile<T, EPI, 8, BN>(o, ep, st);
  }
}

template <typename T, int EPI>
int launch_width(const Operands& o, const EpiArgs<T>& ep, cudaStream_t st) {
  // 32 columns where a quarter of the columns that tiles of 64 compute are padding or more (N up to 32, 65 to 96).  A MiniSTU of 96
  // outputs, 8 x 1000 steps and 24 filters over 64 inputs: 0.572 ms a pass with, 0.597 ms without.
  if constexpr (EPI != EPI_GELU_MUL) {
    if (((long long)o.N + 63) / 64 * 64 * 3 >= ((long long)o.N + 31) / 32 * 32 * 4) return launch_simt<T, EPI, 32>(o, ep, st);
  }
  return launch_simt<T, EPI, 64>(o, ep, st);
}

template <typename T>
int launch_epi(const Operands& o, int epi, const EpiArgs<T>& ep, cudaStream_t st) {
  switch (epi) {
    case EPI_STORE: return launch_width<T, EPI_STORE>(o, ep, st);
    case EPI_RESID: return launch_width<T, EPI_RESID>(o, ep, st);
    case EPI_GELU_MUL: return launch_width<T, EPI_GELU_MUL>(o, ep, st);
    case EPI_HIST: return launch_width<T, EPI_HIST>(o, ep, st);
    case EPI_BLOCKCOL: return launch_width<T, EPI_BLOCKCOL>(o, ep, st);
  }
  return STU_ERR_UNSUPPORTED;
}

}  // namespace

int gemm_simt_dispatch(const void* A, long long lda, const void* B, long long ldb, long long skb, const void* B2,
                       int M, int N, int K, int epi, int causal, const EpiArgsAny& ep, int dtype, cudaStream_t st) {
  const uintptr_t quad = dtype == STU_F32 ? 15 : 7;   // bytes of four elements, less one
  const bool vec_a = lda % 4 == 0 && !((uintptr_t)A & quad);
  const bool vec_b = skb == 1 && ldb % 4 == 0 && !((uintptr_t)B & quad) && !((uintptr_t)B2 & quad);
  const Operands o{A, B, B2, lda, ldb, skb, M, N, K, causal, vec_a, vec_b};
  if (dtype == STU_F32) return launch_epi<float>(o, epi, ep.as<float>(), st);
  if (dtype == STU_BF16) return launch_epi<bf16>(o, epi, ep.as<bf16>(), st);
  return STU_ERR_DTYPE;
}
