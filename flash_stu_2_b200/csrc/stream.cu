// Token-step linear layers for at most 8 activation rows: y[M,N] = epilogue(x[M,K] . W[N,K]^T), the weight read once.
//
// Bound: HBM (the weight), and at these sizes the chain of launches: a 1536 x 1536 projection is 0.7 us of traffic.
// So the kernel is built to have its weights on the way before its input exists.  One CTA per SM owns N / 148
// consecutive output features (no tile granularity: 1536 features are 10 or 11 per CTA); its warps split K and every
// thread copies the 16-byte pieces that it will itself feed to the tensor core (bf16) or its FMAs (fp32) through a
// shared-memory ring of its own with cp.async: no barrier, no staging pass, and the bytes in flight (about 100 KB per
// SM) are bounded by shared memory instead of registers.  The ring is filled ahead of griddepcontrol.wait when the
// caller promises that the weights are nobody's output; shared memory and registers are kept under half an SM so
// that the next launch of the chain can do the same beside this one.
//
// bf16: mma.sync m16n8k16 with the WEIGHTS as the 16-row operand and the rows of x as the 8 columns, the k order
// permuted so that a lane's 16 bytes are its fragment; the partial sums of the 8 warps meet once, at the end.
// fp32: plain FMAs, partial sums folded by a halving butterfly.  Optional fused RMSNorm: statistics while the first
// weights are in flight, every value scaled as the norm kernel would have stored it.
#include "common.cuh"
#include "epilogue.cuh"

int device_sm_count();   // gemm_tc.cu

namespace {

constexpr int NW = 8, THREADS = NW * 32;

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
// 16-byte asynchronous copy; n = 0 fills the slot with zeros and reads nothing
__device__ __forceinline__ void copy16(void* dst, const void* src, unsigned n) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_addr(dst)), "l"(src), "r"(n) : "memory");
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void copy_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
__device__ __forceinline__ void mma_16816(float* c, uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                          uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// Sum of squares of the M <= 8 rows of x, all threads of the CTA on every row; s_part[row][warp] are the partial sums.
template <typename T>
__device__ __forceinline__ void row_squares(const T* __restrict__ x, long long lda, int M, int K, float (*s_part)[NW]) {
  constexpr int V = Elem<T>::VEC;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  float ss[8];
#pragma unroll
  for (int m = 0; m < 8; m++) ss[m] = 0.f;
  for (int k = threadIdx.x * V; k < K; k += THREADS * V) {
#pragma unroll
    for (int m = 0; m < 8; m++)
      if (m < M) {
        float v[V];
        load_vec(x + (size_t)m * lda + k, v);
#pragma unroll
        for (int j = 0; j < V; j++) ss[m] += v[j] * v[j];
      }
  }
#pragma unroll
  for (int m = 0; m < 8; m++)
    if (m < M) {
      const float s = warp_sum(ss[m]);
      if (lane == 0) s_part[m][warp] = s;
    }
}
__device__ __forceinline__ float row_scale(const float* part, int K, float eps) {
  float s = 0.f;
#pragma unroll
  for (int w = 0; w < NW; w++) s += part[w];
  return rsqrtf(s / (float)K + eps);
}

// ------------------------------------------------------------------------------------------------ bf16
// NT tiles of 16 features per step (gate/up: NT/2 of each); D ring stages.  A step is one 32-element chunk of K of one
// group of tiles; warp w takes the chunks w, w + 8, ...
// Shared memory: ring of weights [D][NT][2 halves][256 threads] | ring of x [D][NW][M * 4] | ring of norm weights
// [D][NW][4] | partial sums [NW][NT][4][32] floats (over the ring when there is one group only).
template <int EPI, bool NORM, int NT, int D>
__global__ void __launch_bounds__(THREADS, 2)
    stream_bf16_kernel(const bf16* __restrict__ x, long long lda, const bf16* __restrict__ W, long long ldb,
                       const bf16* __restrict__ W2, int M, int N, int K, EpiArgs<bf16> ep,
                       const bf16* __restrict__ nw, float eps, int early, int groups) {
  constexpr bool DUAL = (EPI == EPI_GELU_MUL);
  constexpr int TF = DUAL ? NT / 2 : NT;   // feature tiles per group
  extern __shared__ uint4 sm[];
  uint4* wring = sm;
  uint4* xring = wring + D * NT * 2 * THREADS;
  uint4* nring = xring + D * NW * M * 4;
  float* red = groups > 1 ? reinterpret_cast<float*>(nring + (NORM ? D * NW * 4 : 0)) : reinterpret_cast<float*>(sm);
  __shared__ float s_part[8][NW];

  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = lane >> 2, q = lane & 3;
  // features of this CTA
  const int r0 = (int)((long long)N * blockIdx.x / gridDim.x), r1 = (int)((long long)N * (blockIdx.x + 1) / gridDim.x);
  const int nchunks = (K + 31) >> 5;
  const int per_warp = warp < nchunks ? (nchunks - warp + NW - 1) / NW : 0;
  const int steps = per_warp * groups;

  auto issue_w = [&](int s) {
    if (s < steps) {
      const int grp = s / per_warp, j = s - grp * per_warp;
      const int k = ((warp + j * NW) << 5) + q * 8;
      const int slot = s % D;
#pragma unroll
      for (int t = 0; t < NT; t++)
#pragma unroll
        for (int h = 0; h < 2; h++) {
          const int r = r0 + (grp * TF + (DUAL ? t % TF : t)) * 16 + h * 8 + g;
          if (r < r1) {   // rows past the end are never stored: what their slots hold does not matter
            const bf16* src = ((DUAL && t >= TF) ? W2 : W) + (size_t)r * ldb;
            const bool ok = k + 8 <= K;
            copy16(wring + ((slot * NT + t) * 2 + h) * THREADS + threadIdx.x, ok ? src + k : src, ok ? 16u : 0u);
          }
        }
      if (NORM && g == 0) {
        const bool ok = k + 8 <= K;
        copy16(nring + (slot * NW + warp) * 4 + q, ok ? nw + k : nw, ok ? 16u : 0u);
      }
    }
    copy_commit();
  };
  auto issue_x = [&](int s) {
    if (s < steps && g < M) {
      const int j = s % per_warp;
      const int k = ((warp + j * NW) << 5) + q * 8;
      const bool ok = k + 8 <= K;
      copy16(xring + ((s % D) * NW + warp) * M * 4 + lane, x + (size_t)g * lda + (ok ? k : 0), ok ? 16u : 0u);
    }
  };

  const bool early_trigger = early && PdlTrigger<EPI>::ahead_of_wait;
  if (early_trigger) pdl_trigger();
  if (!early) pdl_wait();
#pragma unroll
  for (int s = 0; s < D; s++) issue_w(s);
  if (early) pdl_wait();
  if (!early_trigger) pdl_trigger();
#pragma unroll
  for (int s = 0; s < D; s++) {
    issue_x(s);
    copy_commit();
  }
  float r = 0.f;
  if (NORM) {
    row_squares<bf16>(x, lda, M, K, s_part);
    __syncthreads();
    if (g < M) r = row_scale(s_part[g], K, eps);
  }

  float acc[NT][4];
#pragma unroll
  for (int t = 0; t < NT; t++)
#pragma unroll
    for (int i = 0; i < 4; i++) acc[t][i] = 0.f;

  int s = 0;
  for (int grp = 0; grp < groups; grp++) {
    for (int j = 0; j < per_warp; j++, s++) {
      copy_wait<D - 1>();
      const int slot = s % D;
      if (NORM) __syncwarp();   // the norm weights were copied by the lanes of row 0
      uint4 xv = g < M ? xring[(slot * NW + warp) * M * 4 + lane] : make_uint4(0, 0, 0, 0);
      if (NORM) xv = norm_pack(xv, r, nring[(slot * NW + warp) * 4 + q]);
#pragma unroll
      for (int t = 0; t < NT; t++) {
        const uint4 lo = wring[((slot * NT + t) * 2 + 0) * THREADS + threadIdx.x];
        const uint4 hi = wring[((slot * NT + t) * 2 + 1) * THREADS + threadIdx.x];
        mma_16816(acc[t], lo.x, hi.x, lo.y, hi.y, xv.x, xv.y);
        mma_16816(acc[t], lo.z, hi.z, lo.w, hi.w, xv.z, xv.w);
      }
      if (NORM) __syncwarp();   // everybody has read the slot's norm weights
      issue_x(s + D);
      issue_w(s + D);           // commits both
    }
    // ---- the warps' partial sums meet
    if (groups == 1) {
      copy_wait<0>();
      __syncthreads();          // the ring is free
    }
#pragma unroll
    for (int t = 0; t < NT; t++)
#pragma unroll
      for (int i = 0; i < 4; i++) {
        red[((warp * NT + t) * 4 + i) * 32 + lane] = acc[t][i];
        acc[t][i] = 0.f;
      }
    __syncthreads();
    const int rows = min(TF * 16, r1 - (r0 + grp * TF * 16));
    for (int e = threadIdx.x; e < TF * 16 * M; e += THREADS) {
      const int m = e / (TF * 16), f = e - m * (TF * 16);
      if (f < rows) {
        const int t = f >> 4, row = f & 15;
        // row `row`, column m of a tile: lane (row % 8) * 4 + m / 2, register (row / 8) * 2 + m % 2
        const int at = ((row >> 3) * 2 + (m & 1)) * 32 + (row & 7) * 4 + (m >> 1);
        float v = 0.f, v2 = 0.f;
#pragma unroll
        for (int w = 0; w < NW; w++) {
          v += red[(w * NT + t) * 128 + at];
          if (DUAL) v2 += red[(w * NT + TF + t) * 128 + at];
        }
        epilogue_store<bf16, EPI>(ep, m, r0 + grp * TF * 16 + f, v, v2);
      }
    }
    if (groups > 1) __syncthreads();   // the sums have been read
  }
}

template <int EPI, bool NORM, int NT, int D>
int launch_bf16(const bf16* x, long long lda, const bf16* W, long long ldb, const bf16* W2, int M, int N, int K,
                const EpiArgs<bf16>& ep, const bf16* nw, float eps, int early, int grid, int groups, cudaStream_t st) {
  const size_t ring = (size_t)D * (NT * 2 * THREADS + NW * M * 4 + (NORM ? NW * 4 : 0)) * 16;
  const size_t sums = (size_t)NW * NT * 128 * 4;
  const size_t smem = groups > 1 ? ring + sums : (ring > sums ? ring : sums);
  auto k = stream_bf16_kernel<EPI, NORM, NT, D>;
  static SmemLimit limit;
  const cudaError_t granted = allow_smem((const void*)k, 160 * 1024, limit);
  if (granted != cudaSuccess) return (int)granted;
  const cudaError_t e = launch_maybe_overlapped(k, dim3(grid), dim3(THREADS), smem, st, true, x, lda, W, ldb, W2, M, N, K,
                                                ep, nw, eps, early, groups);
  if (e != cudaSuccess) return (int)e;
  STU_CHECK_LAUNCH();
  return STU_OK;
}

// Tiles per step by the features of a CTA; as many ring stages as keep a CTA under half an SM's shared memory.
template <int EPI, bool NORM>
int launch_bf16_tiles(const bf16* x, long long lda, const bf16* W, long long ldb, const bf16* W2, int M, int N, int K,
                      const EpiArgs<bf16>& ep, const bf16* nw, float eps, int early, cudaStream_t st) {
  constexpr bool DUAL = (EPI == EPI_GELU_MUL);
  const int sms = device_sm_count();
  const int grid = N < sms ? N : sms;
  const int rows = (N + grid - 1) / grid;
  const int tiles = (rows + 15) / 16;
#define STU_STREAM(NT_, D_, GROUPS_) \
  return launch_bf16<EPI, NORM, NT_, D_>(x, lda, W, ldb, W2, M, N, K, ep, nw, eps, early, grid, GROUPS_, st)
  if (DUAL) {
    if (tiles == 1) STU_STREAM(2, 5, 1);
    if (tiles == 2) STU_STREAM(4, 2, 1);
    STU_STREAM(6, 2, (tiles + 2) / 3);
  } else {
    if constexpr (!DUAL) {
      if (tiles == 1) STU_STREAM(1, 8, 1);
      if (tiles == 2) STU_STREAM(2, 5, 1);
      if (tiles == 3) STU_STREAM(3, 3, 1);
      if (tiles == 4) STU_STREAM(4, 2, 1);
      STU_STREAM(6, 2, (tiles + 5) / 6);
    }
  }
#undef STU_STREAM
  return STU_ERR_UNSUPPORTED;
}

// ------------------------------------------------------------------------------------------------ fp32
// NR weight rows per step (gate/up: NR/2 of each), MM >= M rows of x, two ring stages.  A step is one 128-element chunk
// of K of one group of rows; wk warps split the chunks, the NW / wk teams of wk warps take the groups in turn.
// Shared memory: ring of weights [2][NR][256] | ring of x [2][M][256] | ring of norm weights [2][256] | partial sums
// [groups][wk][NR * MM] floats.
template <int NV>
__device__ __forceinline__ float fold(float (&v)[NV], int lane) {   // the sum over the warp of v[lane / (32 / NV)]
  int off = 16;
#pragma unroll
  for (int n = NV; n > 1; n >>= 1, off >>= 1) {
#pragma unroll
    for (int i = 0; i < n / 2; i++) {
      const bool up = (lane & off) != 0;
      const float send = up ? v[i] : v[i + n / 2], keep = up ? v[i + n / 2] : v[i];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, send, off);
    }
  }
#pragma unroll
  for (int o = 16 / NV; o > 0; o >>= 1) v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
  return v[0];
}

template <int EPI, bool NORM, int NR, int MM>
__global__ void __launch_bounds__(THREADS, 2)
    stream_f32_kernel(const float* __restrict__ x, long long lda, const float* __restrict__ W, long long ldb,
                      const float* __restrict__ W2, int M, int N, int K, EpiArgs<float> ep,
                      const float* __restrict__ nw, float eps, int early, int wk) {
  constexpr bool DUAL = (EPI == EPI_GELU_MUL);
  constexpr int D = 2, TF = DUAL ? NR / 2 : NR, NV = NR * MM;
  extern __shared__ uint4 sm[];
  uint4* wring = sm;
  uint4* xring = wring + D * NR * THREADS;
  uint4* nring = xring + D * M * THREADS;
  float* red = reinterpret_cast<float*>(nring + (NORM ? D * THREADS : 0));
  __shared__ float s_part[8][NW];

  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int kw = warp % wk, team = warp / wk, teams = NW / wk;
  const int r0 = (int)((long long)N * blockIdx.x / gridDim.x), r1 = (int)((long long)N * (blockIdx.x + 1) / gridDim.x);
  const int ngroups = (r1 - r0 + TF - 1) / TF;
  const int mine = team < ngroups ? (ngroups - team + teams - 1) / teams : 0;
  const int nchunks = (K + 127) >> 7;
  const int per_warp = kw < nchunks ? (nchunks - kw + wk - 1) / wk : 0;
  const int steps = mine * per_warp;

  auto issue_w = [&](int s) {
    if (s < steps) {
      const int gi = s / per_warp, j = s - gi * per_warp;
      const int k = ((kw + j * wk) << 7) + lane * 4;
      const bool ok = k + 4 <= K;
      const int base = r0 + (team + gi * teams) * TF;
#pragma unroll
      for (int i = 0; i < NR; i++) {
        const int r = base + (DUAL ? i % TF : i);
        if (r < r1) {   // rows past the end are never stored
          const float* src = ((DUAL && i >= TF) ? W2 : W) + (size_t)r * ldb;
          copy16(wring + ((s % D) * NR + i) * THREADS + threadIdx.x, ok ? src + k : src, ok ? 16u : 0u);
        }
      }
      if (NORM) copy16(nring + (s % D) * THREADS + threadIdx.x, ok ? nw + k : nw, ok ? 16u : 0u);
    }
    copy_commit();
  };
  auto issue_x = [&](int s) {
    if (s < steps) {
      const int k = ((kw + (s % per_warp) * wk) << 7) + lane * 4;
      const bool ok = k + 4 <= K;
#pragma unroll
      for (int m = 0; m < MM; m++)
        if (m < M) copy16(xring + ((s % D) * M + m) * THREADS + threadIdx.x, x + (size_t)m * lda + (ok ? k : 0), ok ? 16u : 0u);
    }
  };

  const bool early_trigger = early && PdlTrigger<EPI>::ahead_of_wait;
  if (early_trigger) pdl_trigger();
  if (!early) pdl_wait();
#pragma unroll
  for (int s = 0; s < D; s++) issue_w(s);
  if (early) pdl_wait();
  if (!early_trigger) pdl_trigger();
#pragma unroll
  for (int s = 0; s < D; s++) {
    issue_x(s);
    copy_commit();
  }
  float r[MM];
  if (NORM) {
    row_squares<float>(x, lda, M, K, s_part);
    __syncthreads();
#pragma unroll
    for (int m = 0; m < MM; m++) r[m] = m < M ? row_scale(s_part[m], K, eps) : 0.f;
  }

  int s = 0;
  for (int gi = 0; gi < mine; gi++) {
    float acc[NV];
#pragma unroll
    for (int i = 0; i < NV; i++) acc[i] = 0.f;
    for (int j = 0; j < per_warp; j++, s++) {
      copy_wait<D - 1>();
      const int slot = s % D;
      float4 xv[MM];
#pragma unroll
      for (int m = 0; m < MM; m++) {
        xv[m] = m < M ? *reinterpret_cast<const float4*>(xring + (slot * M + m) * THREADS + threadIdx.x)
                      : make_float4(0.f, 0.f, 0.f, 0.f);
        if (NORM) {
          const float4 gw = *reinterpret_cast<const float4*>(nring + slot * THREADS + threadIdx.x);
          xv[m].x = xv[m].x * r[m] * gw.x;
          xv[m].y = xv[m].y * r[m] * gw.y;
          xv[m].z = xv[m].z * r[m] * gw.z;
          xv[m].w = xv[m].w * r[m] * gw.w;
        }
      }
#pragma unroll
      for (int i = 0; i < NR; i++) {
        const float4 w4 = *reinterpret_cast<const float4*>(wring + (slot * NR + i) * THREADS + threadIdx.x);
#pragma unroll
        for (int m = 0; m < MM; m++) {
          float a = acc[i * MM + m];
          a = fmaf(xv[m].x, w4.x, a);
          a = fmaf(xv[m].y, w4.y, a);
          a = fmaf(xv[m].z, w4.z, a);
          acc[i * MM + m] = fmaf(xv[m].w, w4.w, a);
        }
      }
      issue_x(s + D);
      issue_w(s + D);   // commits both
    }
    const float v = fold<NV>(acc, lane);
    if (lane % (32 / NV) == 0) red[((team + gi * teams) * wk + kw) * NV + lane / (32 / NV)] = v;
  }
  __syncthreads();
  for (int e = threadIdx.x; e < (r1 - r0) * M; e += THREADS) {
    const int m = e / (r1 - r0), f = e - m * (r1 - r0);
    const int grp = f / TF, i = f - grp * TF;
    float v = 0.f, v2 = 0.f;
    for (int w = 0; w < wk; w++) {
      v += red[(grp * wk + w) * NV + i * MM + m];
      if (DUAL) v2 += red[(grp * wk + w) * NV + (TF + i) * MM + m];
    }
    epilogue_store<float, EPI>(ep, m, r0 + f, v, v2);
  }
}

template <int EPI, bool NORM, int NR, int MM>
int launch_f32(const float* x, long long lda, const float* W, long long ldb, const float* W2, int M, int N, int K,
               const EpiArgs<float>& ep, const float* nw, float eps, int early, cudaStream_t st) {
  constexpr int TF = (EPI == EPI_GELU_MUL) ? NR / 2 : NR, NV = NR * MM;
  const int nchunks = (K + 127) / 128, sms = device_sm_count();
  // Of the splits over 8 and 4 warps the one that leaves the fewest chunks to the busiest warp: 12 chunks of K over 8 warps
  // take two rounds of which half is idle, over 4 warps of 2 teams three full ones (8 rows: 4608 x 1536 13.4 -> 11.2 us,
  // 50257 x 1536 186 -> 103 with whole rounds of CTAs; 1 row: 4608 x 1536 7.3 -> 6.7).  Beyond three
  // chunks a warp, or over 2 warps, the results' error grows with the sums of a lane (K = 768 over 2 warps: 9.3e-8 for
  // 8.8e-8, 2304 over 4: 1.07e-7 for 1.02e-7).
  int wk = 1, grid = 1, groups = 1, least = 0;
  for (int w = NW; w >= 1; w /= 2) {
    if (w > 1 && w / 2 >= nchunks) continue;
    if (least && (w < 4 || nchunks > 3 * w)) break;
    // one CTA per SM; where its partial sums would need more than 64 KB, rounds of one per SM
    const int max_rows = 65536 / (w * NV * 4) * TF;
    int n = N < sms ? N : sms;
    if ((N + n - 1) / n > max_rows) n = ((N + max_rows - 1) / max_rows + sms - 1) / sms * sms;
    const int gr = ((N + n - 1) / n + TF - 1) / TF, teams = NW / w;
    const int chunks = (n + sms - 1) / sms * ((gr + teams - 1) / teams) * ((nchunks + w - 1) / w);
    if (least == 0 || chunks < least) {
      least = chunks;
      wk = w;
      grid = n;
      groups = gr;
    }
  }
  size_t smem = (size_t)2 * (NR + M + (NORM ? 1 : 0)) * THREADS * 16 + (size_t)groups * wk * NV * 4;
  // 128 rows per SM and more at 5 to 8 rows of x: one CTA per SM for certain.  Where two fit, CTAs that start behind a short
  // kernel pair up on the SMs that are free first and others stay idle (8 rows, 40000 x 768 behind a norm: 70 us for 46)
  if (MM == 8 && N > 128 * sms && smem < 116 * 1024) smem = 116 * 1024;
  auto k = stream_f32_kernel<EPI, NORM, NR, MM>;
  static SmemLimit limit;
  const cudaError_t granted = allow_smem((const void*)k, 200 * 1024, limit);
  if (granted != cudaSuccess) return (int)granted;
  const cudaError_t e = launch_maybe_overlapped(k, dim3(grid), dim3(THREADS), smem, st, true, x, lda, W, ldb, W2, M, N, K,
                                                ep, nw, eps, early, wk);
  if (e != cudaSuccess) return (int)e;
  STU_CHECK_LAUNCH();
  return STU_OK;
}

// Rows per step: eight while the ring then stays under half an SM's shared memory.
template <int EPI, bool NORM>
int launch_f32_rows(const float* x, long long lda, const float* W, long long ldb, const float* W2, int M, int N, int K,
                    const EpiArgs<float>& ep, const float* nw, float eps, int early, cudaStream_t st) {
  if (M == 1) return launch_f32<EPI, NORM, 8, 1>(x, lda, W, ldb, W2, M, N, K, ep, nw, eps, early, st);
  if (M == 2) return launch_f32<EPI, NORM, 8, 2>(x, lda, W, ldb, W2, M, N, K, ep, nw, eps, early, st);
  if (M <= 4) return launch_f32<EPI, NORM, 8, 4>(x, lda, W, ldb, W2, M, N, K, ep, nw, eps, early, st);
  return launch_f32<EPI, NORM, 4, 8>(x, lda, W, ldb, W2, M, N, K, ep, nw, eps, early, st);
}

template <int EPI>
int dispatch_norm(const void* A, long long lda, const void* B, long long ldb, const void* B2, int M, int N, int K,
                  const EpiArgsAny& ep, const void* nw, float eps, int dtype, int early, cudaStream_t st) {
  if (dtype == STU_BF16) {
    const EpiArgs<bf16> e = ep.as<bf16>();
    if (nw)
      return launch_bf16_tiles<EPI, true>((const bf16*)A, lda, (const bf16*)B, ldb, (const bf16*)B2, M, N, K, e,
                                          (const bf16*)nw, eps, early, st);
    return launch_bf16_tiles<EPI, false>((const bf16*)A, lda, (const bf16*)B, ldb, (const bf16*)B2, M, N, K, e,
                                         (const bf16*)nullptr, eps, early, st);
  }
  const EpiArgs<float> e = ep.as<float>();
  if (nw)
    return launch_f32_rows<EPI, true>((const float*)A, lda, (const float*)B, ldb, (const float*)B2, M, N, K, e,
                                      (const float*)nw, eps, early, st);
  return launch_f32_rows<EPI, false>((const float*)A, lda, (const float*)B, ldb, (const float*)B2, M, N, K, e,
                                     (const float*)nullptr, eps, early, st);
}

}  // namespace

// The operands have passed skinny_supported (alignment, K a multiple of the vector width, M <= 64).
// bf16: from 64 KB of weights and 31 features per SM on.  Below that the launch is latency and the 8-feature kernel,
// which keeps nothing in shared memory, is as fast or faster (chain of dependent launches, 1 row: 1536 x 1536 2.9
// against 2.5 us, 1024 x 4096 6.2 against 3.4 us; 8 rows: gate/up 4096 x 1024 a tie), above it this one is (1 row:
// 4608 x 1536 7.4 -> 5.0 us, gate/up 6144 x 1536 14.7 -> 8.6 us = 4.4 TB/s; 8 rows: 8.3 -> 7.1 and 15.9 -> 11.4 us).
// fp32: all (512-wide model, 2 rows: gate/up 6144 x 512 10.6 -> 7.2 us, down 7.8 -> 5.1 us) but the widest gate/up products of
// 5 to 8 rows, which the upkeep of the rings slows down (8 rows with the norm, us, this kernel and the one of skinny.cu
// behind a norm kernel: 4608 x 1536 26.6 and 31.5, 5120 x 1280 29.0 and 26.1, 6144 x 1536 34.6 and 32.0, 9216 x 768 26.3 and 23.2, 12288 x 3072
// 117 and 90) and wide heads of 5 to 8 rows whose K leaves a quarter of the warps idle (8 x 40000 x 768: 70 and 60).  A caller
// that asks for the fused norm gets it, whatever the width.
bool stream_takes(int M, int N, int K, int epi, int dtype, const void* norm_w, bool peer) {
  if (M > 8 || peer || (epi != EPI_STORE && epi != EPI_RESID && epi != EPI_GELU_MUL)) return false;
  if (norm_w && !aligned16(norm_w)) return false;
  const long long sms = device_sm_count();
  if (dtype == STU_F32) {
    if (norm_w || M <= 4) return true;
    if (epi == EPI_GELU_MUL) return N <= 32 * sms;
    const int chunks = (K + 127) / 128, warps = chunks < 3 ? chunks : 4;   // see launch_f32
    return N <= 128 * sms || 5 * chunks > 4 * ((chunks + warps - 1) / warps * warps);
  }
  return N > 30 * sms && (long long)N * K * (epi == EPI_GELU_MUL ? 4 : 2) >= 65536 * sms;
}

int stream_dispatch(const void* A, long long lda, const void* B, long long ldb, const void* B2, int M, int N, int K,
                    int epi, const EpiArgsAny& ep, const void* norm_w, float eps, int dtype, int pdl, cudaStream_t st) {
  const int early = (pdl & STU_FLAG_OVERLAP) ? 1 : 0;
  switch (epi) {
    case EPI_STORE: return dispatch_norm<EPI_STORE>(A, lda, B, ldb, B2, M, N, K, ep, norm_w, eps, dtype, early, st);
    case EPI_RESID: return dispatch_norm<EPI_RESID>(A, lda, B, ldb, B2, M, N, K, ep, norm_w, eps, dtype, early, st);
    case EPI_GELU_MUL: return dispatch_norm<EPI_GELU_MUL>(A, lda, B, ldb, B2, M, N, K, ep, norm_w, eps, dtype, early, st);
  }
  return STU_ERR_UNSUPPORTED;
}
