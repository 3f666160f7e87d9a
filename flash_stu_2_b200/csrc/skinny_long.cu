// Token-step linears of up to 8 rows over long rows of weights (bf16): y = x[M,K] @ W[N,K]^T, store and residual epilogues
// (the contraction of the features of all filters, flash_stu/modules/stu.py:100-118, mini_stu/stu_lds.py:338-394: K = filters * d).
//
// Bound: the weights, once, from HBM.  The kernel of 8 features per CTA (skinny.cu) reads the activation rows in every CTA, as many
// bytes from L2 as there are weights, and asks for a round of loads only when the last one is used up.  Here a CTA owns 32 features, K is
// split over a cluster (the sums meet in distributed shared memory, added in rank order), and every lane keeps a ring of its own
// operands under way (cp.async into slots that no other thread reads: no barrier in the loop).  Fragments as in skinny.cu: 16 bytes of a
// weight row and of an activation row per lane and chunk of 32, the k order permuted alike in both.
#include <cooperative_groups.h>

#include <atomic>

#include "common.cuh"
#include "epilogue.cuh"

namespace cg = cooperative_groups;

int device_sm_count();   // gemm_tc.cu

namespace {

constexpr int NT = 4;   // n-tiles (8 features each) per CTA
constexpr int NW = 8;   // warps, taking the chunks in turn
constexpr int SLOT = 32 * 16;

__device__ __forceinline__ void mma_16816(float* c, uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void copy16(uint32_t dst, const bf16* src, bool in) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(in ? 16 : 0) : "memory");
}
__device__ __forceinline__ uint4 own_slot(uint32_t at) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(at) : "memory");
  return v;
}

constexpr int ST = 8;                    // chunks under way per warp
constexpr int STAGE = (NT + 1) * SLOT;
constexpr int SMEM_BYTES = NW * ST * STAGE;

template <int EPI, int KS>
__global__ void __launch_bounds__(NW * 32) skinny_long_kernel(const bf16* __restrict__ x, long long lda, const bf16* __restrict__ W,
                                                              long long ldb, int M, int N, int K, EpiArgs<bf16> ep, int pdl) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, q = lane & 3;
  const int n0 = blockIdx.x * (8 * NT);
  const int chunks = (K + 31) >> 5, per = (chunks + KS - 1) / KS;
  const int c0 = (KS > 1 ? (int)blockIdx.y * per : 0) + warp, c_end = KS > 1 ? min(chunks, ((int)blockIdx.y + 1) * per) : chunks;
  const uint32_t ring = (uint32_t)__cvta_generic_to_shared(smem) + warp * ST * STAGE + lane * 16;
  const bf16* wrow[NT];
#pragma unroll
  for (int j = 0; j < NT; j++) wrow[j] = W + (size_t)min(n0 + 8 * j + g, N - 1) * ldb + q * 8;   // (features past N: the last one, not stored)
  auto load_w = [&](int st, int c) {
    const bool in = c < c_end && (c << 5) + q * 8 + 8 <= K;
#pragma unroll
    for (int j = 0; j < NT; j++) copy16(ring + st * STAGE + j * SLOT, in ? wrow[j] + (c << 5) : W, in);
  };
  auto load_x = [&](int st, int c) {
    const bool in = c < c_end && (c << 5) + q * 8 + 8 <= K;
    const bool row = in && g < M;
    copy16(ring + st * STAGE + NT * SLOT, row ? x + (size_t)g * lda + (c << 5) + q * 8 : x, row);
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  if (pdl & STU_FLAG_EARLY_TRIGGER) pdl_trigger();
#pragma unroll
  for (int st = 0; st < ST; st++) load_w(st, c0 + st * NW);   // (under STU_FLAG_OVERLAP beside the kernel in front)
  pdl_wait();
  if (!(pdl & STU_FLAG_EARLY_TRIGGER)) pdl_trigger();
#pragma unroll
  for (int st = 0; st < ST; st++) load_x(st, c0 + st * NW);

  float acc[NT][4];
#pragma unroll
  for (int j = 0; j < NT; j++)
#pragma unroll
    for (int i = 0; i < 4; i++) acc[j][i] = 0.f;
  int st = 0;
  for (int c = c0; c < c_end; c += NW) {
    asm volatile("cp.async.wait_group %0;" ::"n"(ST - 1) : "memory");
    uint4 wv[NT];
#pragma unroll
    for (int j = 0; j < NT; j++) wv[j] = own_slot(ring + st * STAGE + j * SLOT);
    const uint4 xv = own_slot(ring + st * STAGE + NT * SLOT);
    __syncwarp();   // mma.sync takes the whole warp
#pragma unroll
    for (int j = 0; j < NT; j++) {
      mma_16816(acc[j], xv.x, 0u, xv.y, 0u, wv[j].x, wv[j].y);   // rows 8..15 are zero
      mma_16816(acc[j], xv.z, 0u, xv.w, 0u, wv[j].z, wv[j].w);
    }
    load_w(st, c + ST * NW);
    load_x(st, c + ST * NW);
    if (++st == ST) st = 0;
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();   // every ring is used up: its place is taken by the sums
  float* red = reinterpret_cast<float*>(smem);   // [NW][NT][4][32]
  float* part = red + NW * NT * 128;             // [8 rows][8 NT features]
#pragma unroll
  for (int j = 0; j < NT; j++)
#pragma unroll
    for (int i = 0; i < 4; i++) red[((warp * NT + j) * 4 + i) * 32 + lane] = acc[j][i];
  __syncthreads();
  // element (row, col) of n-tile j lies in lane row * 4 + col / 2, register col % 2
  for (int e = threadIdx.x; e < NT * 64; e += NW * 32) {
    const int row = e / (8 * NT), f = e % (8 * NT), j = f >> 3, col = f & 7;
    const int at = (j * 4 + (col & 1)) * 32 + row * 4 + (col >> 1);
    float s = 0.f;
#pragma unroll
    for (int w = 0; w < NW; w++) s += red[w * NT * 128 + at];
    part[e] = s;
  }
  cg::cluster_group cluster = cg::this_cluster();
  if constexpr (KS > 1) cluster.sync(); else __syncthreads();
  const int rank = KS > 1 ? (int)cluster.block_rank() : 0;
  constexpr int SHARE = NT * 64 / KS;   // of this CTA
  for (int e = rank * SHARE + threadIdx.x; e < (rank + 1) * SHARE; e += NW * 32) {
    const int m = e / (8 * NT), n = n0 + e % (8 * NT);
    float s = 0.f;
#pragma unroll
    for (int r = 0; r < KS; r++) s += KS > 1 ? *cluster.map_shared_rank(part + e, r) : part[e];
    if (m < M && n < N) epilogue_store<bf16, EPI>(ep, m, n, s, 0.f);
  }
  if constexpr (KS > 1) cluster.sync();   // the other CTAs' sums stay alive until read
}

template <int EPI, int KS>
int launch_long(const void* A, long long lda, const void* B, long long ldb, int M, int N, int K, const EpiArgs<bf16>& ep, int pdl,
                cudaStream_t st) {
  auto kern = skinny_long_kernel<EPI, KS>;
  static SmemLimit limit;
  cudaError_t e = allow_smem((const void*)kern, SMEM_BYTES, limit);
  if (e != cudaSuccess) return (int)e;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((N + 8 * NT - 1) / (8 * NT), KS);
  cfg.blockDim = dim3(NW * 32);
  cfg.dynamicSmemBytes = SMEM_BYTES;
  cfg.stream = st;
  cudaLaunchAttribute at[2];
  int n = 0;
  if (KS > 1) {
    at[n].id = cudaLaunchAttributeClusterDimension;
    at[n].val.clusterDim.x = 1;
    at[n].val.clusterDim.y = KS;
    at[n++].val.clusterDim.z = 1;
  }
  if ((pdl & STU_FLAG_OVERLAP) && pdl_enabled()) {
    at[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[n++].val.programmaticStreamSerializationAllowed = 1;
  }
  cfg.attrs = at;
  cfg.numAttrs = n;
  e = cudaLaunchKernelEx(&cfg, kern, (const bf16*)A, lda, (const bf16*)B, ldb, M, N, K, ep, pdl);
  if (e != cudaSuccess) return (int)e;
  STU_CHECK_LAUNCH();
  return STU_OK;
}

// Whether the GPU holds this many clusters of KS CTAs at a time (the SMs of a GPC are no multiple of 4)
template <int KS>
bool clusters_fit(int clusters) {
  static std::atomic<int> known[STU_MAX_DEVICES] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= STU_MAX_DEVICES) dev = 0;
  int n = known[dev].load(std::memory_order_relaxed);
  if (n > 0) return clusters <= n;
  auto kern = skinny_long_kernel<EPI_STORE, KS>;
  static SmemLimit limit;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(1, KS);
  cfg.blockDim = dim3(NW * 32);
  cfg.dynamicSmemBytes = SMEM_BYTES;
  cudaLaunchAttribute at;
  at.id = cudaLaunchAttributeClusterDimension;
  at.val.clusterDim.x = at.val.clusterDim.z = 1;
  at.val.clusterDim.y = KS;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  if (allow_smem((const void*)kern, SMEM_BYTES, limit) != cudaSuccess || cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess) {
    (void)cudaGetLastError();
    return false;
  }
  known[dev].store(n, std::memory_order_relaxed);
  return clusters <= n;
}

template <int EPI>
int launch_long_split(int ks, const void* A, long long lda, const void* B, long long ldb, int M, int N, int K, const EpiArgs<bf16>& ep,
                      int pdl, cudaStream_t st) {
  switch (ks) {
    case 1: return launch_long<EPI, 1>(A, lda, B, ldb, M, N, K, ep, pdl, st);
    case 2: return launch_long<EPI, 2>(A, lda, B, ldb, M, N, K, ep, pdl, st);
    default: return launch_long<EPI, 4>(A, lda, B, ldb, M, N, K, ep, pdl, st);
  }
}

}  // namespace

// Up to 8 rows of 4096 weights and more, where the kernels of 8 features per CTA would need a second wave (from 4104 weights or 16 features per SM
// on) or there are 9.4 M weights and more and the clusters of four run at a time (B200: up to 33 of them, N = 1056; in two waves 4 x 1128 x
// 8368 took 13.7 us where those kernels take 8.6).  us, 8 rows, those kernels and this one: 1024 x 49152 26.7 and 21.5, 768 x 24576 17.3 and 10.7, 768 x 12288
// 12.1 and 7.0, 1024 x 12288 8.5 and 8.0, 1024 x 8192 6.6 and 6.8, 1024 x 4096 3.7 and 4.4, 512 x 49152 15.5 and 16.0, 1280 x 5120 9.1 and 5.9, 2048 x 4096 7.3
// and 7.8, 2048 x 8192 11.9 and 9.2, 4096 x 16384 39 and 25 (1 and 4 rows alike).
bool skinny_long_takes(int M, int N, int K, int epi, bool norm, bool peer) {
  const int sms = device_sm_count();
  if (M > 8 || (epi != EPI_STORE && epi != EPI_RESID) || norm || peer || K < 4096 || N > 32 * sms) return false;
  if (N > 8 * sms) return K > 4096 || N > 16 * sms;
  return N >= 640 && (long long)N * K >= 9400000 && clusters_fit<4>((N + 8 * NT - 1) / (8 * NT));
}

int skinny_long_dispatch(const void* A, long long lda, const void* B, long long ldb, int M, int N, int K, int epi, const EpiArgs<bf16>& ep,
                         int pdl, cudaStream_t st) {
  // K is split until there is about one CTA per SM (1536 x 8192: one CTA per tile 9.6 us, two 8.2, four 10.8), in clusters that run at a time
  const int ctas = (N + 8 * NT - 1) / (8 * NT);
  const int ks = clusters_fit<4>(ctas) ? 4 : clusters_fit<2>(ctas) ? 2 : 1;
  if (epi == EPI_STORE) return launch_long_split<EPI_STORE>(ks, A, lda, B, ldb, M, N, K, ep, pdl, st);
  return launch_long_split<EPI_RESID>(ks, A, lda, B, ldb, M, N, K, ep, pdl, st);
}
