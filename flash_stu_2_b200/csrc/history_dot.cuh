// Dot products of 8 sequences' histories with their channel's reversed taps, as the kernels that stream histories take them
// (stu_decode_pipe, stu_block_step, stu_stream_ahead: one order of operations, the same bits): a unit of SEG positions of 8 sequences
// x 8 channels and their taps lies in shared memory, a warp takes one channel, and the products are the diagonal of mma.sync m16n8k16
// products with the history as A and the taps as B.
#pragma once
#include "common.cuh"
#include "tma.cuh"

constexpr int SEG = 256;                       // history positions per unit
constexpr int HIST_BYTES = 64 * SEG * 2;       // 8 sequences x 8 channels x SEG bf16
constexpr int TAP_BYTES = 8 * SEG * 2;
constexpr int HIST_STAGE_BYTES = HIST_BYTES + TAP_BYTES;

__device__ __forceinline__ uint4 lds128(const void* p) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "r"(tma::smem_u32(p)));
  return v;
}
__device__ __forceinline__ void mma16816(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                         uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// rows 8..15 of the A tile are zero
__device__ __forceinline__ void mma_rows8(float (&c)[4], const uint4& a, const uint4& b) {
  mma16816(c, a.x, 0u, a.y, 0u, b.x, b.y);
  mma16816(c, a.z, 0u, a.w, 0u, b.z, b.w);
}
// keep the first `keep` (1..7) of the eight bf16 values of a vector
__device__ __forceinline__ uint4 keep_first(const uint4& v, int keep) {
  uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
  for (int j = 0; j < 4; j++)
    if (2 * j + 1 >= keep) w[j] = (2 * j < keep) ? (w[j] & 0x0000ffffu) : 0u;
  return make_uint4(w[0], w[1], w[2], w[3]);
}

// One unit of a warp's channel ch, added to its four accumulators.  `left`: positions from the unit's first on that are stored
// history; looked at in the last unit alone (tail).
__device__ __forceinline__ void history_unit(float (&acc)[4][4], const unsigned char* stage, int ch, int lane, bool tail, int left) {
  const int g = lane >> 2, q = lane & 3;
  const bf16* H = reinterpret_cast<const bf16*>(stage) + (size_t)(g * 8 + ch) * SEG;
  const bf16* T = reinterpret_cast<const bf16*>(stage + HIST_BYTES) + (size_t)ch * SEG;
#pragma unroll
  for (int win = 0; win < SEG / 64; win++) {
#pragma unroll
    for (int pass = 0; pass < 2; pass++) {
      // row g takes the chunks of its 64-value window in the order that keeps the eight lanes of a
      // quarter warp (two rows x four chunks) on distinct banks; taps use the same order, only D[g][g] is read
      const int koff = win * 64 + ((q + 4 * ((g & 1) ^ pass)) << 3);
      uint4 a = lds128(H + koff);
      const uint4 b = lds128(T + koff);
      if (tail) {
        const int keep = left - koff;   // values of this vector that are stored history
        if (keep <= 0) a = make_uint4(0, 0, 0, 0);
        else if (keep < 8) a = keep_first(a, keep);
      }
      mma_rows8(acc[win], a, b);
    }
  }
}
// D[g][g] sits in the lane with q = g / 2, register g & 1: whether this lane holds a sum, and the sum of sequence g.
__device__ __forceinline__ bool history_lane(int lane) { return (lane & 3) == (lane >> 3); }
__device__ __forceinline__ float history_sum(const float (&acc)[4][4], int lane) {
  const float even = (acc[0][0] + acc[1][0]) + (acc[2][0] + acc[3][0]);
  const float odd = (acc[0][1] + acc[1][1]) + (acc[2][1] + acc[3][1]);
  return (lane >> 2) & 1 ? odd : even;
}
