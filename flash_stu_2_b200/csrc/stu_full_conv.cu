// Full variant, fp32, short calls (the others: stu_full_conv_f32_umma.cu): the operand U of the contraction for all K filters in one launch
// (flash_stu/modules/stu.py:100-118; MiniSTU mini_stu/stu.py:240-269):
//   U+-[b,t,k,i] = E +- Q,   E = sum_{j even} phi[j,k] x[b,t-j,i],   Q the same over odd j.
//
// Bound: FMA issue.  Filter by filter (Toeplitz matrices, three GEMMs with them, a combine pass) this was 120 launches
// of 3 to 16 us for 24 filters, E and Q went through memory, and a triangle's empty half was computed tile by tile.
// Here a CTA owns 64 time indices m (t = 2m and 2m + 1) of 4 * TX channels under one filter, a thread 4 x 4 of them with
// four sums each: E and Q of both parities share the inputs xe[s] = x[2s], xo[s] = x[2s+1] and their taps
//   E_even += f[2(m-s)] xe[s]   E_odd += f[2(m-s)] xo[s]   Q_odd += f[2(m-s)+1] xe[s]   Q_even += f[2(m-s)-1] xo[s].
// Two channels at a time (fma.rn.f32x2: inputs are pairs as they lie, taps are staged twice), which takes half the issue slots;
// a thread's taps slide by one as s advances, so a step of s is 32 such instructions, two 16-byte reads of the inputs and two 8-byte
// ones of the taps.  Sums over s run in order, as the GEMMs' did.  24 filters, 8 x 1000 positions of 64 channels: 1.35 ms; one product
// at a time, 64 channels a CTA, copies' addresses worked out for every step 0.40; in pairs at 32 channels (three CTAs per SM) 0.36;
// addresses once and all long sums ahead of all short ones 0.32; the 32 steps unrolled, so that the sliding costs no moves,
// 0.28 (42 TFLOP/s of the causal half; the pairs' issue rate alone would be 0.20).
#include "common.cuh"

namespace {

typedef unsigned long long f32x2;   // two fp32 values of one register pair
__device__ __forceinline__ f32x2 pair_of(float lo, float hi) { return (f32x2)__float_as_uint(hi) << 32 | __float_as_uint(lo); }
__device__ __forceinline__ float half_of(f32x2 v, int hi) { return __uint_as_float((uint32_t)(hi ? v >> 32 : v)); }
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}

constexpr int MT = 64, ST = 32;   // time indices per CTA, inputs per step of the pipeline

template <int TX>
__global__ void __launch_bounds__(TX * 16, 24 / TX) full_conv_kernel(const float* __restrict__ hist, int Lh,
                                                            const float* __restrict__ phi, int L, int K,
                                                            float* __restrict__ U, long long ldU, int rows, int d,
                                                            int both, int t0, int t_end, int tiles_m) {
  constexpr int CT = TX * 4, THREADS = TX * 16, PX = CT + 4;
  constexpr int QX = 2 * CT * ST / 4 / THREADS;    // 16-byte pieces of the inputs per thread and step
  constexpr int NT = 2 * (MT + ST);                // taps per step: even ones, odd ones
  constexpr int QT = (NT + THREADS - 1) / THREADS;
  static_assert(QX * 4 * THREADS == 2 * CT * ST, "thread layout");
  __shared__ __align__(16) float xs[2][2][ST][PX];   // [buffer][parity][s][channel]
  __shared__ f32x2 taps[2][NT];                      // each twice: both halves of an operand
  const int tid = threadIdx.x, tx = tid % TX, ty = tid / TX;
  // one dimension holds any number of tiles; the longest sums of all channels and filters first
  const unsigned per_tile = gridDim.x / (unsigned)tiles_m, at = blockIdx.x % per_tile;
  const int k = at % K, c0 = at / K * CT;
  const int tm = tiles_m - 1 - (int)(blockIdx.x / per_tile);
  const int m0 = (t0 >> 1) + tm * MT;
  const int s_end = min(m0 + MT, (t_end + 1) >> 1);  // inputs that some output of the tile needs

  // this thread's pieces: one channel, QX times four inputs; QT taps
  float rx[QX][4], rt[QT];
  const bool mine = c0 + tid % CT < rows;
  const float* src[QX];
  int from[QX], tap_at[QT];
  const float* tap[QT];
#pragma unroll
  for (int i = 0; i < QX; i++) {
    const int q = (tid + i * THREADS) / CT, p = q / (ST / 4);
    from[i] = 2 * (q % (ST / 4) * 4) + p;   // time of the first of the four inputs, less 2 s0
    src[i] = hist + ((size_t)(c0 + (mine ? tid % CT : 0)) * 2 + p) * Lh + q % (ST / 4) * 4;
  }
#pragma unroll
  for (int i = 0; i < QT; i++) {   // even[e] = f[2 (m0 - s0 - ST + e)], odd[e] = f[2 (m0 - s0 - ST + e) + 1]
    const int e = tid + i * THREADS, odd = e >= MT + ST;
    tap_at[i] = e < NT ? 2 * (m0 - ST + e - odd * (MT + ST)) + odd : -1;
    tap[i] = phi + (long long)tap_at[i] * K + k;
  }
  auto fetch = [&](int s0) {
    if (2 * (s0 + ST) <= t_end) {   // (rows of the history are 16-byte aligned)
#pragma unroll
      for (int i = 0; i < QX; i++) {
        const float4 v = mine ? *reinterpret_cast<const float4*>(src[i] + s0) : make_float4(0.f, 0.f, 0.f, 0.f);
        rx[i][0] = v.x; rx[i][1] = v.y; rx[i][2] = v.z; rx[i][3] = v.w;
      }
    } else {
#pragma unroll
      for (int i = 0; i < QX; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) rx[i][j] = (mine && from[i] + 2 * (s0 + j) < t_end) ? src[i][s0 + j] : 0.f;
    }
#pragma unroll
    for (int i = 0; i < QT; i++) {
      const int j = tap_at[i] - 2 * s0;
      rt[i] = (j >= 0 && j < L) ? *(tap[i] - 2ll * s0 * K) : 0.f;
    }
  };
  auto stage = [&](int buf) {
#pragma unroll
    for (int i = 0; i < QX; i++) {
      const int e = tid + i * THREADS, c = e % CT, q = e / CT;
#pragma unroll
      for (int j = 0; j < 4; j++) xs[buf][q / (ST / 4)][q % (ST / 4) * 4 + j][c] = rx[i][j];
    }
#pragma unroll
    for (int i = 0; i < QT; i++)
      if (tid + i * THREADS < NT) taps[buf][tid + i * THREADS] = pair_of(rt[i], rt[i]);
  };

  f32x2 ee[4][2], eo[4][2], qo[4][2], qe[4][2];   // [m][pair of channels]
#pragma unroll
  for (int i = 0; i < 4; i++)
#pragma unroll
    for (int j = 0; j < 2; j++) ee[i][j] = eo[i][j] = qo[i][j] = qe[i][j] = 0;

  fetch(0);
  stage(0);
  __syncthreads();
  for (int s0 = 0, buf = 0; s0 < s_end; s0 += ST, buf ^= 1) {
    const bool more = s0 + ST < s_end;
    if (more) fetch(s0 + ST);
    // taps of m = m0 + 4 ty + i against s = s0 + u: even[ST + 4 ty + i - u], odd the same index and the one below
    const f32x2* te = taps[buf] + ST + 4 * ty;
    const f32x2* to = te + MT + ST;
    f32x2 t4[4], o[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
      t4[i] = te[i];
      o[i] = to[i];
    }
#pragma unroll
    for (int u = 0; u < ST; u++) {
      const f32x2 below = to[-1 - u];
      const ulonglong2 ve = *reinterpret_cast<const ulonglong2*>(&xs[buf][0][u][tx * 4]);
      const ulonglong2 vo = *reinterpret_cast<const ulonglong2*>(&xs[buf][1][u][tx * 4]);
      const f32x2 xe[2] = {ve.x, ve.y}, xo[2] = {vo.x, vo.y};
      const f32x2 od[5] = {below, o[0], o[1], o[2], o[3]};
#pragma unroll
      for (int i = 0; i < 4; i++) {
#pragma unroll
        for (int j = 0; j < 2; j++) ee[i][j] = fma2(t4[i], xe[j], ee[i][j]);
#pragma unroll
        for (int j = 0; j < 2; j++) eo[i][j] = fma2(t4[i], xo[j], eo[i][j]);
#pragma unroll
        for (int j = 0; j < 2; j++) qe[i][j] = fma2(od[i], xo[j], qe[i][j]);
#pragma unroll
        for (int j = 0; j < 2; j++) qo[i][j] = fma2(od[i + 1], xe[j], qo[i][j]);
      }
      t4[3] = t4[2]; t4[2] = t4[1]; t4[1] = t4[0]; t4[0] = te[-1 - u];
      o[3] = o[2]; o[2] = o[1]; o[1] = o[0]; o[0] = below;
    }
    if (more) stage(buf ^ 1);   // last read before the barrier of the step before
    __syncthreads();
  }

  const int c = c0 + tx * 4;
  const bool vec = d % 4 == 0 && ldU % 4 == 0 && (reinterpret_cast<uintptr_t>(U) & 15) == 0;
#pragma unroll
  for (int i = 0; i < 4; i++)
#pragma unroll
    for (int p = 0; p < 2; p++) {
      const int t = 2 * (m0 + ty * 4 + i) + p;
      if (t < t0 || t >= t_end) continue;
      float up[4], um[4];
#pragma unroll
      for (int j = 0; j < 4; j++) {
        const float E = half_of(p ? eo[i][j >> 1] : ee[i][j >> 1], j & 1), Q = half_of(p ? qo[i][j >> 1] : qe[i][j >> 1], j & 1);
        up[j] = E + Q;
        um[j] = E - Q;
      }
      if (vec) {
        if (c < rows) {   // four channels of one sequence
          float* at = U + ((size_t)(c / d) * (t_end - t0) + (t - t0)) * ldU + (size_t)k * d + c % d;
          *reinterpret_cast<float4*>(at) = make_float4(up[0], up[1], up[2], up[3]);
          if (both) *reinterpret_cast<float4*>(at + (size_t)K * d) = make_float4(um[0], um[1], um[2], um[3]);
        }
      } else {
#pragma unroll
        for (int j = 0; j < 4; j++)
          if (c + j < rows) {
            float* at = U + ((size_t)((c + j) / d) * (t_end - t0) + (t - t0)) * ldU + (size_t)k * d + (c + j) % d;
            at[0] = up[j];
            if (both) at[(size_t)K * d] = um[j];
          }
      }
    }
}

}  // namespace

// hist: [B*d][2][Lh] holding the inputs of times [0, t_end); phi: [L][K]; U: rows (b, t - t0) of ldU elements, column
// sign*K*d + k*d + i.  fp32 only (bf16 products belong on the tensor cores).
extern "C" int stu_full_conv(const void* hist, int Lh, const void* phi, int L, int K, void* U, long long ldU, int B, int d,
                             int both_signs, int t0, int t_end, int dtype, void* stream) {
  if (!hist || !phi || !U) return STU_ERR_NULL;
  if (B <= 0 || d <= 0 || K <= 0 || K > 65535 || L <= 0 || t0 < 0 || t_end <= t0 || t_end > 2 * Lh ||
      ldU < (long long)(both_signs ? 2 : 1) * K * d)
    return STU_ERR_SHAPE;
  if (dtype != STU_F32) return STU_ERR_DTYPE;
  if (Lh % 4 || !aligned16(hist)) return STU_ERR_ALIGN;
  const long long rows = (long long)B * d;
  const int tiles_m = (((t_end + 1) >> 1) - (t0 >> 1) + MT - 1) / MT;
  const int ct = rows <= 16 ? 16 : 32;   // channels per CTA
  const long long ctas = (rows + ct - 1) / ct * K * tiles_m;
  if (rows > (1 << 21) || ctas > 0x7fffffffll) return STU_ERR_UNSUPPORTED;   // the grid (its outputs would be 500 GB)
  cudaStream_t st = (cudaStream_t)stream;
  // 32 channels per CTA, 16 where half of them would be padding (narrow layers of one sequence)
#define STU_FULL_CONV(TX_)                                                                                         \
  full_conv_kernel<TX_><<<(unsigned)ctas, TX_ * 16, 0, st>>>(                                                      \
      (const float*)hist, Lh, (const float*)phi, L, K, (float*)U, ldU, (int)rows, d, both_signs, t0, t_end, tiles_m)
  if (ct == 16) STU_FULL_CONV(4);
  else STU_FULL_CONV(8);
#undef STU_FULL_CONV
  STU_CHECK_LAUNCH();
  return STU_OK;
}
