// Full variant, fp32: the operand U of the contraction for all K filters in one launch
// (flash_stu/modules/stu.py:100-118; MiniSTU mini_stu/stu.py:240-269):
//   U+-[b,t,k,i] = E +- Q,   E = sum_{j even} phi[j,k] x[b,t-j,i],   Q the same over odd j.
//
// Bound: FFMA issue.  Filter by filter (Toeplitz matrices, three GEMMs with them, a combine pass) this was 120 launches
// of 3 to 16 us for 24 filters, E and Q went through memory, and a triangle's empty half was computed tile by tile.
// Here a CTA owns 64 time indices m (t = 2m and 2m + 1) of 4 * TX channels under one filter, a thread 4 x 4 of them with
// four sums each: E and Q of both parities share the inputs xe[s] = x[2s], xo[s] = x[2s+1] and their taps
//   E_even += f[2(m-s)] xe[s]   E_odd += f[2(m-s)] xo[s]   Q_odd += f[2(m-s)+1] xe[s]   Q_even += f[2(m-s)-1] xo[s].
// A thread's taps slide by one as s advances, so a step of s costs 64 FMAs, two 16-byte reads of the inputs and two
// words of taps.  Sums over s run in order, as the GEMMs' did.  24 filters, 8 x 1000 positions of 64 channels: 1.35 -> 0.40 ms
// (29 TFLOP/s of the causal half).
#include "common.cuh"

namespace {

constexpr int MT = 64, ST = 32;   // time indices per CTA, inputs per step of the pipeline

template <int TX>
__global__ void __launch_bounds__(TX * 16, 32 / TX) full_conv_kernel(const float* __restrict__ hist, int Lh,
                                                            const float* __restrict__ phi, int L, int K,
                                                            float* __restrict__ U, long long ldU, int rows, int d,
                                                            int both, int t0, int t_end, int tiles_m) {
  constexpr int CT = TX * 4, THREADS = TX * 16, PX = CT + 4;
  constexpr int QX = 2 * CT * ST / 4 / THREADS;    // 16-byte pieces of the inputs per thread and step
  constexpr int NT = 2 * (MT + ST);                // taps per step: even ones, odd ones
  constexpr int QT = (NT + THREADS - 1) / THREADS;
  static_assert(QX * 4 * THREADS == 2 * CT * ST, "thread layout");
  __shared__ __align__(16) float xs[2][2][ST][PX];   // [buffer][parity][s][channel]
  __shared__ float taps[2][NT];
  const int tid = threadIdx.x, tx = tid % TX, ty = tid / TX;
  const int k = blockIdx.z, c0 = blockIdx.y * CT;
  const int tm = tiles_m - 1 - (int)blockIdx.x;      // the longest sums first
  const int m0 = (t0 >> 1) + tm * MT;
  const int s_end = min(m0 + MT, (t_end + 1) >> 1);  // inputs that some output of the tile needs

  float rx[QX][4], rt[QT];
  auto fetch = [&](int s0) {
#pragma unroll
    for (int i = 0; i < QX; i++) {
      const int e = tid + i * THREADS, c = e % CT, q = e / CT, p = q / (ST / 4), s = s0 + q % (ST / 4) * 4;
      const float* src = hist + ((size_t)(c0 + c) * 2 + p) * Lh + s;
      if (c0 + c < rows && 2 * (s + 3) + p < t_end) {   // (rows of the history are 16-byte aligned)
        const float4 v = *reinterpret_cast<const float4*>(src);
        rx[i][0] = v.x; rx[i][1] = v.y; rx[i][2] = v.z; rx[i][3] = v.w;
      } else {
#pragma unroll
        for (int j = 0; j < 4; j++) rx[i][j] = (c0 + c < rows && 2 * (s + j) + p < t_end) ? src[j] : 0.f;
      }
    }
#pragma unroll
    for (int i = 0; i < QT; i++) {   // even[e] = f[2 (m0 - s0 - ST + e)], odd[e] = f[2 (m0 - s0 - ST + e) + 1]
      const int e = tid + i * THREADS, odd = e >= MT + ST;
      const int j = 2 * (m0 - s0 - ST + e - odd * (MT + ST)) + odd;
      rt[i] = (e < NT && j >= 0 && j < L) ? phi[(size_t)j * K + k] : 0.f;
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
      if (tid + i * THREADS < NT) taps[buf][tid + i * THREADS] = rt[i];
  };

  float ee[4][4], eo[4][4], qo[4][4], qe[4][4];   // [m][channel]
#pragma unroll
  for (int i = 0; i < 4; i++)
#pragma unroll
    for (int j = 0; j < 4; j++) ee[i][j] = eo[i][j] = qo[i][j] = qe[i][j] = 0.f;

  fetch(0);
  stage(0);
  __syncthreads();
  for (int s0 = 0, buf = 0; s0 < s_end; s0 += ST, buf ^= 1) {
    const bool more = s0 + ST < s_end;
    if (more) fetch(s0 + ST);
    // taps of m = m0 + 4 ty + i against s = s0 + u: even[ST + 4 ty + i - u], odd the same index and the one below
    const float* te = taps[buf] + ST + 4 * ty;
    const float* to = te + MT + ST;
    float t4[4], o[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
      t4[i] = te[i];
      o[i] = to[i];
    }
#pragma unroll 4
    for (int u = 0; u < ST; u++) {
      const float below = to[-1 - u];
      float xe[4], xo[4];
      *reinterpret_cast<float4*>(xe) = *reinterpret_cast<const float4*>(&xs[buf][0][u][tx * 4]);
      *reinterpret_cast<float4*>(xo) = *reinterpret_cast<const float4*>(&xs[buf][1][u][tx * 4]);
      const float od[5] = {below, o[0], o[1], o[2], o[3]};
      // (four in a row share the tap: its register is read once; with them interleaved a MiniSTU pass took 0.624 ms, so 0.597)
#pragma unroll
      for (int i = 0; i < 4; i++) {
#pragma unroll
        for (int j = 0; j < 4; j++) ee[i][j] = fmaf(t4[i], xe[j], ee[i][j]);
#pragma unroll
        for (int j = 0; j < 4; j++) eo[i][j] = fmaf(t4[i], xo[j], eo[i][j]);
#pragma unroll
        for (int j = 0; j < 4; j++) qe[i][j] = fmaf(od[i], xo[j], qe[i][j]);
#pragma unroll
        for (int j = 0; j < 4; j++) qo[i][j] = fmaf(od[i + 1], xe[j], qo[i][j]);
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
        const float E = p ? eo[i][j] : ee[i][j], Q = p ? qo[i][j] : qe[i][j];
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
  if (rows > (1 << 21)) return STU_ERR_UNSUPPORTED;   // the grid's second dimension
  const int tiles_m = (((t_end + 1) >> 1) - (t0 >> 1) + MT - 1) / MT;
  cudaStream_t st = (cudaStream_t)stream;
  // 64 channels per CTA; fewer where the last tile would be mostly padding (narrow layers of one sequence)
#define STU_FULL_CONV(TX_)                                                                                         \
  full_conv_kernel<TX_><<<dim3(tiles_m, (unsigned)((rows + 4 * TX_ - 1) / (4 * TX_)), K), TX_ * 16, 0, st>>>(      \
      (const float*)hist, Lh, (const float*)phi, L, K, (float*)U, ldU, (int)rows, d, both_signs, t0, t_end, tiles_m)
  if (rows <= 16) STU_FULL_CONV(4);
  else if (rows <= 32) STU_FULL_CONV(8);
  else STU_FULL_CONV(16);
#undef STU_FULL_CONV
  STU_CHECK_LAUNCH();
  return STU_OK;
}
