// Cached token step of the full STU variant, everything before the contraction with M_phi in one kernel (bf16, up to 32
// filters): RMSNorm, append, the K even-tap and K odd-tap sums over the whole history, U+- = E +- Q, position
// (flash_stu/modules/stu.py:100-118 for the new position t = 2 sn + p only; the reference has no cached STU step).
//
//   E[(b,i), k] = sum_{s<=sn} phi[2(sn-s), k] hist[b,i,p][s],      Q[(b,i), k] = sum_s phi[2(sn-s)+-1, k] hist[b,i,1-p][s]
//
// Bound: the history, both parities, once.  It is streamed straight into mma.sync fragments (16 channels x 32 positions of a
// row per pair of 16-byte loads, the k order permuted so that a lane's 16 bytes are its fragment); the taps come from the
// reversed table in its eight alignments (ops.taps_rev8: every 8 taps an aligned load), a few of them per position of 16 or
// 32 channels, from L1 and L2.  A CTA owns 16 * MT channels of one sequence; its 8 warps take the 32-position chunks in
// turn, their sums meet in shared memory.  As a kernel that rebuilt the K x Lh tap matrices, a GEMM against them (both
// tap sets for both parities) and a kernel each to combine and to advance, behind the norm kernel, this was 5 launches: 8
// sequences of 1024 channels near position 2800, the whole layer step, replayed from a graph, 63.6 us; this form 55.9 (layer
// prefill and 64 steps 8.42 -> 7.94 ms).  ops.full_decode_step_pays says where that form stays the faster one, ops.full_decode_step_tc5_pays
// where the kernel of stu_full_step_umma.cu is.
#include "common.cuh"

int device_sm_count();   // gemm_tc.cu

namespace {

constexpr int NW = 8, THREADS = NW * 32;

__device__ __forceinline__ void mma_16816(float* c, uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint4 stream16(const bf16* p) {   // read once
  uint4 v;
  asm volatile("ld.global.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}
// the first n of eight values, zeros behind them
__device__ __forceinline__ uint4 first_of(uint4 v, int n) {
  uint32_t* w = reinterpret_cast<uint32_t*>(&v);
#pragma unroll
  for (int i = 0; i < 4; i++) w[i] = n >= 2 * i + 2 ? w[i] : (n == 2 * i + 1 ? w[i] & 0xffffu : 0u);
  return v;
}

// NT: tiles of 8 filters; MT: tiles of 16 channels.  taps: [8][2K][Lh + 8], even taps of the K filters, then odd taps.
template <int NT, int MT>
__global__ void __launch_bounds__(THREADS, 2)
    full_step_kernel(const bf16* __restrict__ x, long long x_rstride, const bf16* __restrict__ nw, float eps,
                     bf16* __restrict__ hist, const bf16* __restrict__ taps, int* __restrict__ pos, bf16* __restrict__ U,
                     int B, int d, int K, int Lh, int limit, int both, int* __restrict__ status) {
  constexpr int CH = 16 * MT;
  extern __shared__ float red[];   // [NW][MT][2][NT][4][32]
  __shared__ float s_part[NW], s_xn[CH], s_tap0[8 * NT];
  __shared__ int s_t;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, q = lane & 3;
  const int per_seq = (d + CH - 1) / CH, b = blockIdx.x / per_seq, i0 = (blockIdx.x - b * per_seq) * CH;
  const size_t pitch = (size_t)Lh + 8;
  pdl_wait();
  pdl_trigger();
  if (tid == 0) {
    const int t = *(volatile int*)pos;
    s_t = t;
    if (t >= 0 && t < limit) {
      // the last CTA that has read the position moves it on
      __threadfence();
      if (atomicAdd(&pos[1], 1) == (int)gridDim.x - 1) {
        pos[1] = 0;
        for (int i = 0; i < B; i++)
          if (pos[2 * i] >= 0 && pos[2 * i] < 2 * Lh) pos[2 * i] += 1;
      }
    } else if (blockIdx.x == 0 && status) {
      atomicExch(status, 2);
    }
  }
  const bf16* xr = x + (size_t)b * x_rstride;
  uint4 xv = make_uint4(0, 0, 0, 0);   // the row's first piece of this thread, on its way beside the history
  if (nw && tid * 8 < d) xv = *reinterpret_cast<const uint4*>(xr + tid * 8);
  __syncthreads();
  const int t = s_t;
  if (t < 0 || t >= limit) return;
  const int p = t & 1, sn = t >> 1;
  const int cnt[2] = {sn, p ? sn + 1 : sn};   // history entries of the two sums (E: without the new input)
  const bf16 *hbase[2], *tbase[2];
  int hoff[MT][2], toff[NT];
#pragma unroll
  for (int a = 0; a < 2; a++) {
    const int o = a == 0 ? Lh - 1 - sn : Lh - cnt[1], al = o & 7;
    hbase[a] = hist + ((size_t)((size_t)b * d + i0) * 2 + (p ^ a)) * Lh;
    tbase[a] = taps + ((size_t)al * 2 + a) * K * pitch + (o - al);
  }
#pragma unroll
  for (int mt = 0; mt < MT; mt++)
#pragma unroll
    for (int h = 0; h < 2; h++) hoff[mt][h] = min(mt * 16 + h * 8 + g, d - 1 - i0) * 2 * Lh;   // channels past d: any row
#pragma unroll
  for (int n = 0; n < NT; n++) toff[n] = min(n * 8 + g, K - 1) * (int)pitch;
  float acc[2][MT][NT][4];
#pragma unroll
  for (int a = 0; a < 2; a++)
#pragma unroll
    for (int mt = 0; mt < MT; mt++)
#pragma unroll
      for (int n = 0; n < NT; n++)
#pragma unroll
        for (int c = 0; c < 4; c++) acc[a][mt][n][c] = 0.f;
  const int nch = (cnt[1] + 31) >> 5;   // cnt[1] >= cnt[0]
#pragma unroll (MT == 1 && NT <= 3 ? 2 : 1)
  for (int c = warp; c < nch; c += NW) {
    const int s = c * 32 + q * 8;
    uint4 hv[2][MT][2], tv[2][NT];
#pragma unroll
    for (int a = 0; a < 2; a++) {
      const bool in = s < cnt[a];
#pragma unroll
      for (int mt = 0; mt < MT; mt++)
#pragma unroll
        for (int h = 0; h < 2; h++) hv[a][mt][h] = in ? stream16(hbase[a] + hoff[mt][h] + s) : make_uint4(0, 0, 0, 0);
#pragma unroll
      for (int n = 0; n < NT; n++) tv[a][n] = in ? __ldg(reinterpret_cast<const uint4*>(tbase[a] + toff[n] + s)) : make_uint4(0, 0, 0, 0);
    }
#pragma unroll
    for (int a = 0; a < 2; a++) {
      if (s + 8 > cnt[a]) {   // past the position: whatever the cache holds there
#pragma unroll
        for (int mt = 0; mt < MT; mt++)
#pragma unroll
          for (int h = 0; h < 2; h++) hv[a][mt][h] = first_of(hv[a][mt][h], cnt[a] - s);
      }
      __syncwarp();
#pragma unroll
      for (int mt = 0; mt < MT; mt++)
#pragma unroll
        for (int n = 0; n < NT; n++) {
          const uint4 &lo = hv[a][mt][0], &hi = hv[a][mt][1], &w = tv[a][n];
          mma_16816(acc[a][mt][n], lo.x, hi.x, lo.y, hi.y, w.x, w.y);
          mma_16816(acc[a][mt][n], lo.z, hi.z, lo.w, hi.w, w.z, w.w);
        }
    }
  }
#pragma unroll
  for (int a = 0; a < 2; a++)
#pragma unroll
    for (int mt = 0; mt < MT; mt++)
#pragma unroll
      for (int n = 0; n < NT; n++)
#pragma unroll
        for (int c = 0; c < 4; c++) red[((((warp * MT + mt) * 2 + a) * NT + n) * 4 + c) * 32 + lane] = acc[a][mt][n][c];
  // ---- the new input of this CTA's channels, normalised as the norm kernel would have stored it
  float r = 1.f;
  if (nw) {
    float ss = 0.f;
    for (int v = tid; v * 8 < d; v += THREADS) {
      if (v != tid) xv = *reinterpret_cast<const uint4*>(xr + v * 8);
      float f[8];
      load_vec(reinterpret_cast<const bf16*>(&xv), f);
#pragma unroll
      for (int j = 0; j < 8; j++) ss += f[j] * f[j];
    }
    ss = warp_sum(ss);
    if (lane == 0) s_part[warp] = ss;
    __syncthreads();
    ss = 0.f;
#pragma unroll
    for (int w = 0; w < NW; w++) ss += s_part[w];
    r = rsqrtf(ss / (float)d + eps);
  }
  // (the taps at distance 0: behind the wait, since the kernel in front may have just written them)
  if (tid >= THREADS - 8 * NT) {
    const int k = tid - (THREADS - 8 * NT);
    s_tap0[k] = Elem<bf16>::to_f(taps[(size_t)min(k, K - 1) * pitch + Lh - 1]);
  }
  if (tid < CH && i0 + tid < d) {
    const float v = Elem<bf16>::to_f(xr[i0 + tid]);
    const bf16 xn = nw ? __float2bfloat16_rn(v * r * Elem<bf16>::to_f(nw[i0 + tid])) : xr[i0 + tid];
    s_xn[tid] = Elem<bf16>::to_f(xn);
    hist[((size_t)((size_t)b * d + i0 + tid) * 2 + p) * Lh + sn] = xn;
  }
  __syncthreads();
  bf16* urow = U + (size_t)b * (both ? 2 : 1) * K * d + i0;
  for (int e = tid; e < CH * K; e += THREADS) {
    const int c = e % CH, k = e / CH;
    if (i0 + c >= d) continue;
    // channel c, filter k of a tile: lane (c % 8) * 4 + (k % 8) / 2, register (c % 16) / 8 * 2 + k % 2
    const int at = (((c >> 3) & 1) * 2 + (k & 1)) * 32 + (c & 7) * 4 + ((k & 7) >> 1);
    float E = 0.f, Q = 0.f;
#pragma unroll
    for (int w = 0; w < NW; w++) {
      const float* m = red + (((w * MT + (c >> 4)) * 2) * NT + (k >> 3)) * 128 + at;
      E += m[0];
      Q += m[NT * 128];
    }
    E = round_to<bf16>(E + s_xn[c] * s_tap0[k]);
    Q = round_to<bf16>(Q);
    urow[(size_t)k * d + c] = __float2bfloat16_rn(E + Q);
    if (both) urow[(size_t)(K + k) * d + c] = __float2bfloat16_rn(E - Q);
  }
}

template <int NT, int MT>
int launch_step(const bf16* x, long long xs, const bf16* nw, float eps, bf16* hist, const bf16* taps, int* pos, bf16* U, int B,
                int d, int K, int Lh, int limit, int both, int* status, cudaStream_t st) {
  const size_t smem = (size_t)NW * MT * 2 * NT * 128 * 4;
  auto k = full_step_kernel<NT, MT>;
  static SmemLimit lim;
  cudaError_t e = allow_smem((const void*)k, smem, lim);
  if (e != cudaSuccess) return (int)e;
  const int grid = B * ((d + 16 * MT - 1) / (16 * MT));
  e = launch_maybe_overlapped(k, dim3(grid), dim3(THREADS), smem, st, true, x, xs, nw, eps, hist, taps, pos, U, B, d, K, Lh,
                              limit, both, status);
  if (e != cudaSuccess) return (int)e;
  STU_CHECK_LAUNCH();
  return STU_OK;
}

}  // namespace

// x [B][d] (row stride x_rstride): the layer's residual rows with norm_w, else the normalised rows.  taps8 [8][2K][Lh+8]:
// stu_taps_rev8 of the even taps of the K filters and of their odd taps.  U [B][(2 or 1) K d].  Positions [0, limit).
extern "C" int stu_full_decode_step(const void* x, long long x_rstride, const void* norm_w, float eps, void* hist, const void* taps8,
                                    int* pos, void* U, int B, int d, int K, int Lh, int limit, int both_signs, int* status,
                                    int dtype, void* stream) {
  if (!x || !hist || !taps8 || !pos || !U) return STU_ERR_NULL;
  if (B <= 0 || d <= 0 || K <= 0 || Lh <= 0 || limit <= 0 || limit > 2 * Lh) return STU_ERR_SHAPE;
  if (dtype != STU_BF16) return STU_ERR_DTYPE;
  if (K > 32) return STU_ERR_UNSUPPORTED;
  if (Lh % 8 || !aligned16(hist) || !aligned16(taps8)) return STU_ERR_ALIGN;
  if (norm_w && (d % 8 || x_rstride % 8 || !aligned16(x))) return STU_ERR_ALIGN;
  const bf16 *xp = (const bf16*)x, *np = (const bf16*)norm_w, *tp = (const bf16*)taps8;
  cudaStream_t st = (cudaStream_t)stream;
  // 32 channels per CTA (the taps are read half as often) while that leaves no SM without one and the sums fit the registers.  us,
  // 32 and 16 channels, 24 filters, position 1000: 192 CTAs of 32 (4 x 1536) 10.1 and 13.1, 128 (4 x 1024) 8.5 and 7.7; position
  // 3000: 256 (8 x 1024) 16.3 and 20.4, 384 (12 x 1024) 32.0 and 32.2.
  const bool wide = (long long)B * ((d + 31) / 32) >= device_sm_count();
#define STU_STEP(NT_, MT_) \
  return launch_step<NT_, MT_>(xp, x_rstride, np, eps, (bf16*)hist, tp, pos, (bf16*)U, B, d, K, Lh, limit, both_signs, status, st)
  switch ((K + 7) / 8) {
    case 1:
      if (wide) STU_STEP(1, 2);
      STU_STEP(1, 1);
    case 2:
      if (wide) STU_STEP(2, 2);
      STU_STEP(2, 1);
    case 3:
      if (wide) STU_STEP(3, 2);
      STU_STEP(3, 1);
    default: STU_STEP(4, 1);
  }
#undef STU_STEP
}
