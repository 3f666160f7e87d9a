// Token steps of larger batches with the history streams taken off the chain.
//
// An approx STU layer's sum over the history for position t + 1 reads the other time parity than position t writes: it needs
// nothing that step t produces.  stu_stream_ahead_kernel computes these sums for ALL layers of a model as one launch beside the step's
// chain of small products, on a few SMs that it has to itself, and stu_stream_finish_kernel, in the chain, adds the new token's
// own term to what the launch of the step before left:
//   part[layer][(t + 1) & 1][b][c] = sum_{i < s} hist[b][c][p][i] * tap_c[s - i]          s = (t + 1) >> 1, p = (t + 1) & 1
//   hist[b][c][t & 1][t >> 1] = xp ; out = x + round(2 * (part[layer][t & 1] + xp * tap_c[0])) ; xn = rmsnorm(out) * norm_w
// (the arithmetic of stu_decode_pipe_kernel and of the norm kernel, in their order: the same bits).
//
// Control words ctl[4] of a step's buffers: the position that the next launch computes, arrived CTAs, the positions that the two
// halves of part hold.
#include "common.cuh"
#include "history_dot.cuh"
#include "tma.cuh"

namespace {

constexpr int STAGES = 6;                      // 216 KB: the SM is this CTA's alone, and so are its loads in flight
constexpr int STAGE_BYTES = HIST_STAGE_BYTES;
constexpr int GROUPS = 2;                      // of 8 consumer warps, each with a row of its own
constexpr int NTHREADS = (8 * GROUPS + 1) * 32;   // and 1 producer warp
constexpr int MAX_LAYERS = 64;

struct LayerMaps {
  CUtensorMap hist, taps;
};
struct AheadParams {
  LayerMaps maps[MAX_LAYERS];
  float* part;   // [layers][2][B][d]
  int* ctl;
  int* status;
  int layers, B, d, Lh;
};


// A row is 8 sequences x 8 channels of a layer; CTA i owns rows i, i + grid, ... of all layers.  As in stu_decode_pipe_kernel a unit of
// 256 positions arrives by two bulk tensor copies, warp w takes channel w, and the dot products are the diagonal of mma.sync products.
__global__ void __launch_bounds__(NTHREADS, 1) stu_stream_ahead_kernel(const __grid_constant__ AheadParams P) {
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + STAGES * STAGE_BYTES);
  uint64_t* empty_bar = full_bar + STAGES;
  __shared__ int s_abort, s_issued;
  volatile int* abort_flag = &s_abort;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2;
  const int G = gridDim.x, B = P.B, d = P.d, Lh = P.Lh;
  const int ncg = d >> 3, rows = ((B + 7) >> 3) * ncg, total = rows * P.layers;
  if (tid == 0) {
    for (int i = 0; i < STAGES; i++) {
      tma::mbar_init(&full_bar[i], 1);
      tma::mbar_init(&empty_bar[i], 8);
    }
    s_abort = 0;
    s_issued = 0;
    tma::fence_barrier_init();
  }
  const int t = *(volatile const int*)P.ctl;
  __syncthreads();
  const bool inside = t >= 0 && t < 2 * Lh;   // (behind the last position of the capacity there is nothing to prepare)
  const int p = t & 1, s = inside ? t >> 1 : 0, nsl = (s + SEG - 1) / SEG;
  if (warp == 8 * GROUPS) {
    const bool leader = elect_one();
    const int o = Lh - 1 - s, e = o & 7, xo = o - e;   // reversed tap row of position s at its 16-byte alignment
    int n = 0, st = 0;
    uint32_t ph = 1;
    bool ok = true;
    for (int r0 = blockIdx.x; ok && r0 < total; r0 += GROUPS * G)
      for (int sl = 0; ok && sl < nsl; sl++)
        for (int r = r0; r < min(r0 + GROUPS * G, total); r += G, n++) {   // the groups' rows in turn
          const int layer = r / rows, rr = r - layer * rows, bg = rr / ncg, cg = rr - bg * ncg;
          ok = tma::warp_wait_bounded(&empty_bar[st], ph, abort_flag);
          if (!ok) break;
          if (leader) {
            unsigned char* dst = smem + st * STAGE_BYTES;
            tma::mbar_expect_tx(&full_bar[st], STAGE_BYTES);
            tma::load_4d(dst, &P.maps[layer].hist, &full_bar[st], sl * SEG, p, cg * 8, bg * 8);
            tma::load_3d(dst + HIST_BYTES, &P.maps[layer].taps, &full_bar[st], xo + sl * SEG, cg * 8, e);
          }
          __syncwarp();
          if (++st == STAGES) st = 0, ph ^= 1u;
        }
    if (leader) s_issued = n;
  } else {
    const int ch = warp & 7, group = warp >> 3;
    int n0 = 0;   // units ahead of this round of rows
    bool ok = true;
    for (int r0 = blockIdx.x; ok && r0 < total; r0 += GROUPS * G) {
      const int r = r0 + group * G, here = min(GROUPS, (total - r0 + G - 1) / G);   // rows of this round
      if (r >= total) break;
      const int layer = r / rows, rr = r - layer * rows, bg = rr / ncg, cg = rr - bg * ncg;
      float acc[4][4];
#pragma unroll
      for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) acc[i][j] = 0.f;
      for (int sl = 0; sl < nsl; sl++) {
        const int n = n0 + sl * here + group, st = n % STAGES;
        ok = tma::warp_wait_bounded(&full_bar[st], (uint32_t)(n / STAGES) & 1u, abort_flag);
        if (!ok) break;
        history_unit(acc, smem + st * STAGE_BYTES, ch, lane, sl == nsl - 1, s - sl * SEG);
        __syncwarp();
        if (lane == 0) tma::mbar_arrive(&empty_bar[st]);
      }
      n0 += nsl * here;
      if (ok && inside && history_lane(lane) && bg * 8 + g < B)
        P.part[((size_t)(layer * 2 + p) * B + bg * 8 + g) * d + cg * 8 + ch] = history_sum(acc, lane);
    }
  }
  __syncthreads();
  if (s_abort && tid == 0) {
    if (P.status) atomicExch(P.status, 7);
    const int issued = s_issued;   // copies that were issued but never consumed must land before shared memory is released
    for (int n = issued > STAGES ? issued - STAGES : 0; n < issued; n++) {
      int dummy = 0;
      tma::mbar_wait_bounded(&full_bar[n % STAGES], ((uint32_t)(n / STAGES)) & 1u, &dummy);
    }
  }
  // the last CTA to finish says which position is there, and moves on; after a wait that ran out the sums stay unannounced
  if (tid == 0) {
    __threadfence();
    if (s_abort) atomicExch(&P.ctl[2 + p], -1);
    if (atomicAdd(&P.ctl[1], 1) == G - 1) {
      if (inside && !s_abort) atomicCAS(&P.ctl[2 + p], t - 2, t);
      P.ctl[1] = 0;
      P.ctl[0] = t + 1;
    }
  }
}

struct FinishParams {
  const bf16 *x, *xp, *taps8, *norm_w;
  bf16 *hist, *out, *xn;
  const float* part;   // of this layer: [2][B][d]
  const int* ctl;
  int* pos;
  int* status;
  int B, d, Lh, overlap;
  float eps;
};

// One CTA per sequence: the new token's term, the residual, the append and the norm behind them.  Under STU_FLAG_OVERLAP everything that
// the step before left (sums, taps, position) is read ahead of the wait for the projection: the caller's word that no kernel
// which may still be under way writes it (the steps of a replayed graph, which begin when the replay before is complete).
__global__ void __launch_bounds__(128) stu_stream_finish_kernel(const FinishParams P) {
  constexpr int NV = 4;   // vectors of 8 channels per thread: d up to 4096
  const int b = blockIdx.x, d = P.d, Lh = P.Lh;
  const size_t LP = (size_t)Lh + 8;
  if (P.overlap) pdl_trigger();
  const int t = P.pos[2 * b], p = t & 1, s = t >> 1;
  const bool ok = t >= 0 && t < 2 * Lh && P.ctl[2 + p] == t;
  float y[NV][8], w0[NV][8];
  if (ok) {
#pragma unroll
    for (int v = 0; v < NV; v++) {
      const int c = (v * 128 + threadIdx.x) * 8;
      if (c < d) {
        const float* pr = P.part + ((size_t)p * P.B + b) * d + c;
        load_vec(pr, y[v]);
        load_vec(pr + 4, y[v] + 4);
#pragma unroll
        for (int j = 0; j < 8; j++) w0[v][j] = __bfloat162float(P.taps8[(size_t)(c + j) * LP + (Lh - 1)]);
      }
    }
  }
  pdl_wait();   // the projection is the kernel before this one
  if (!P.overlap) pdl_trigger();
  if (!ok) {
    if (threadIdx.x == 0 && P.status) atomicExch(P.status, t < 0 || t >= 2 * Lh ? 2 : 8);
    return;
  }
  float ss = 0.f;
#pragma unroll
  for (int v = 0; v < NV; v++) {
    const int c = (v * 128 + threadIdx.x) * 8;
    if (c < d) {
      float xp[8], x[8];
      const uint4 raw = *reinterpret_cast<const uint4*>(P.xp + (size_t)b * d + c);
      load_vec(reinterpret_cast<const bf16*>(&raw), xp);
      load_vec(P.x + (size_t)b * d + c, x);
#pragma unroll
      for (int j = 0; j < 8; j++) {
        P.hist[((size_t)((size_t)b * d + c + j) * 2 + p) * Lh + s] = reinterpret_cast<const bf16*>(&raw)[j];
        y[v][j] = round_to<bf16>(x[j] + round_to<bf16>(2.f * __fadd_rn(y[v][j], __fmul_rn(xp[j], w0[v][j]))));
        ss += y[v][j] * y[v][j];
      }
      store_vec(P.out + (size_t)b * d + c, y[v]);
    }
  }
  __shared__ float red[4];
  ss = warp_sum(ss);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = ss;
  __syncthreads();   // (every thread has read the position as well)
  if (threadIdx.x == 0) P.pos[2 * b] = t + 1;
  const float r = rsqrtf((red[0] + red[1] + red[2] + red[3]) / (float)d + P.eps);
#pragma unroll
  for (int v = 0; v < NV; v++) {
    const int c = (v * 128 + threadIdx.x) * 8;
    if (c < d) {
      float g[8];
      load_vec(P.norm_w + c, g);
#pragma unroll
      for (int j = 0; j < 8; j++) g[j] = y[v][j] * r * g[j];
      store_vec(P.xn + (size_t)b * d + c, g);
    }
  }
}

}  // namespace

extern "C" int stu_stream_ahead(const void* const* hist, const void* const* taps8, int layers, float* part, int* ctl, int B, int d,
                                int Lh, int sms, int* status, int dtype, void* stream) {
  if (!hist || !taps8 || !part || !ctl) return STU_ERR_NULL;
  if (layers <= 0 || B <= 0 || d <= 0 || Lh <= 0 || sms <= 0 || d % 8 || Lh % 8) return STU_ERR_SHAPE;
  if (dtype != STU_BF16 || layers > MAX_LAYERS) return STU_ERR_UNSUPPORTED;
  static_assert(sizeof(AheadParams) <= 32764, "kernel parameters");
  AheadParams P;
  for (int i = 0; i < layers; i++) {
    if (!hist[i] || !taps8[i]) return STU_ERR_NULL;
    if (!aligned16(hist[i]) || !aligned16(taps8[i])) return STU_ERR_ALIGN;
    const cuuint64_t dims[4] = {(cuuint64_t)Lh, 2, (cuuint64_t)d, (cuuint64_t)B};
    const cuuint64_t strides[3] = {(cuuint64_t)Lh * 2, (cuuint64_t)Lh * 4, (cuuint64_t)d * Lh * 4};
    const cuuint32_t box[4] = {SEG, 1, 8, 8};
    int rc = tma::encode_bf16(&P.maps[i].hist, hist[i], 4, dims, strides, box);
    if (rc != STU_OK) return rc;
    const cuuint64_t LP = (cuuint64_t)Lh + 8;
    const cuuint64_t tdims[3] = {LP, (cuuint64_t)d, 8};
    const cuuint64_t tstrides[2] = {LP * 2, (cuuint64_t)d * LP * 2};
    const cuuint32_t tbox[3] = {SEG, 8, 1};
    if ((rc = tma::encode_bf16(&P.maps[i].taps, taps8[i], 3, tdims, tstrides, tbox)) != STU_OK) return rc;
  }
  P.part = part;
  P.ctl = ctl;
  P.status = status;
  P.layers = layers;
  P.B = B;
  P.d = d;
  P.Lh = Lh;
  const size_t smem = (size_t)STAGES * STAGE_BYTES + 2 * STAGES * sizeof(uint64_t) + 1024;
  static SmemLimit limit;
  const cudaError_t e = allow_smem((const void*)stu_stream_ahead_kernel, smem, limit);
  if (e != cudaSuccess) return (int)e;
  const long long rows = (long long)layers * ((B + 7) / 8) * (d / 8);
  stu_stream_ahead_kernel<<<(int)(rows < sms ? rows : sms), NTHREADS, smem, (cudaStream_t)stream>>>(P);
  STU_CHECK_LAUNCH();
  return STU_OK;
}

extern "C" int stu_stream_finish(const void* x, const void* xp, void* hist, const void* taps8, int* pos, const float* part,
                                 const int* ctl, const void* norm_w, float eps, void* out, void* xn, int B, int d, int Lh,
                                 int* status, int dtype, void* stream) {
  if (!x || !xp || !hist || !taps8 || !pos || !part || !ctl || !norm_w || !out || !xn) return STU_ERR_NULL;
  const bool overlap = (dtype & STU_FLAG_OVERLAP) != 0;
  dtype &= ~STU_FLAG_OVERLAP;
  if (B <= 0 || d <= 0 || Lh <= 0 || d % 8 || Lh % 8) return STU_ERR_SHAPE;
  if (dtype != STU_BF16 || d > 4096) return STU_ERR_UNSUPPORTED;
  if (!aligned16(x) || !aligned16(xp) || !aligned16(part) || !aligned16(norm_w) || !aligned16(out) || !aligned16(xn)) return STU_ERR_ALIGN;
  FinishParams P{(const bf16*)x, (const bf16*)xp, (const bf16*)taps8, (const bf16*)norm_w, (bf16*)hist, (bf16*)out, (bf16*)xn,
                 part, ctl, pos, status, B, d, Lh, overlap ? 1 : 0, eps};
  const cudaError_t e = launch_maybe_overlapped(stu_stream_finish_kernel, dim3(B), dim3(128), 0, (cudaStream_t)stream, overlap, P);
  if (e != cudaSuccess) return (int)e;
  STU_CHECK_LAUNCH();
  return STU_OK;
}
