// Prefill convolutions of the full STU variant in fp32 on the 5th-generation tensor cores, all filters in one launch
// (flash_stu/modules/stu.py:100-118; MiniSTU mini_stu/stu.py:240-269).
//
//   U+-[b,t,k,i] = E +- Q,   E = sum_{j even} phi[j,k] x[b,t-j,i],   Q the same over odd j.
//
// The Toeplitz products of stu_full_conv_umma.cu: per filter and tap set a table of 8 x 8 core matrices, of which 23 consecutive ones
// are a 128 x 64 block in the un-swizzled K-major operand layout (the A operand, rows are positions in descending groups of
// eight), times rows of the parity-split history (the B operand).  Taps and history come as three bf16 parts each (split3.cuh, one
// kernel in front), six products of parts make an fp32 product, an accumulator takes 64 positions and is then added to fp32 sums in
// registers, since the tensor core's own sums are not rounded to nearest; E and Q of a tile stay in registers.
//
// Bound: L2, from which a stage of 24 instructions (66 cycles each at 128 channels) takes 57 KB: 1.4 us a stage on all SMs are 6 TB/s.  24
// filters, the CUDA-core kernel (stu_full_conv.cu) and this one, us: 8 x 1000 positions of 64 channels 277 and 101, 4 x 600 of 512 478 and 200, 16
// filters, 8 x 2048 of 96 1074 and 276 (stu_full_conv_f32_tc5_pays says where that one stays the faster).  Error against float64: 3.3e-7 and
// 9.6e-8, 2.6e-7 and 9.1e-8, 4.7e-7 and 1.1e-7 (32 positions per accumulator: the same, and twice the reads of tensor memory, 121 us for the first).
//
// Roles (one persistent CTA per SM, 320 threads): warp 0 producer, warp 1 MMA issuer, warps 2-9 sums and outputs (a quarter of the
// rows and half of the channels each).  Tiles run from the latest positions (the most work) down, the filters of a channel block side by
// side, so that its history rows are read from L2.  Sums that are not finite are computed again on the CUDA cores, a warp's part of a
// tile at a time: values that are not finite, or above 2^87, have no such parts, and sums above 2^79 overflow.  24 filters, 8 x 1000 positions of 64
// channels, all of them, 2.2 ms (a thread's chain for each, 39 ms; the CUDA-core kernel 0.29), with one NaN in a channel 0.8 (7.9).
// Every load is a plain single-CTA copy of this GPU's own memory.  Every wait is bounded: on expiry the CTA raises status 9, lets issued
// copies land (bounded), frees its tensor memory and returns.
#include <cuda.h>

#include <algorithm>

#include "common.cuh"
#include "split3.cuh"
#include "tma.cuh"

int device_sm_count();

namespace {

constexpr int BM = 128, BK = 64;
constexpr int A_ENTRIES = 23;                  // core matrices of a 128 x 64 block: q' + kc = 0 .. 15 + 7
constexpr int CM = 3 * 128;                    // bytes from one core matrix to the next: the three parts of each lie together
constexpr int A_BYTES = A_ENTRIES * CM, A_PITCH = 9216;
constexpr int STAGES = 3, ACCS = 4;
constexpr int EPI_WARPS = 8, THREADS = 64 + 32 * EPI_WARPS;
constexpr int SROW = 36, STG_BYTES = 32 * SROW * 4;  // a warp's staging block of 32 positions x 32 channels
constexpr int STATUS_CONV_WAIT = 9;

struct Ctl {
  uint64_t full[STAGES], empty[STAGES], acc_full[ACCS], acc_empty[ACCS];
  uint32_t tmem_slot;
  int abort_flag, issued, consumed;
};
static_assert(sizeof(Ctl) <= 256, "control block");

template <int TN> __host__ __device__ constexpr int plane_b() { return TN * BK * 2; }
template <int TN> __host__ __device__ constexpr int stages_bytes() { return STAGES * (3 * plane_b<TN>() + A_PITCH); }
template <int TN> constexpr int smem_bytes() { return stages_bytes<TN>() + EPI_WARPS * STG_BYTES + 256 + 1024; }
static_assert(smem_bytes<128>() <= 227 * 1024, "shared memory");

struct Geom {
  int B, d, K, L, Lh, Tn, t0, t_end;
  int both;               // U- too
  int mb_first, nb;       // 128-position blocks with outputs: mb_first .. nb - 1
  int n_ct;               // channel tiles
  int entries;            // table entries per filter and tap set
  int Lp;                 // positions of a row of the history's parts
  long long ldU;
};

// Tap sets: 0 even taps, 1 odd taps of outputs of parity 1 from inputs of parity 0, 2 odd taps the other way round.
__device__ __forceinline__ int tap_of(int kind, int dist) { return 2 * dist + (kind == 0 ? 0 : (kind == 1 ? 1 : -1)); }
__host__ __device__ inline int table_entries(int nb) { return 16 * (nb - 1) + 31; }

// The parts of the taps, tab[k][kind][e][part][r][w]: the tap at distance 120 - 8 X + r - w, X = e - 16 (nb - 1), zero above the diagonal
// and past the filter; and of the history, planes[part][row][p][s], zero past the call's last position.  A thread per 8 values of either.
__global__ void __launch_bounds__(256) full_conv_parts_kernel(const float* __restrict__ phi, const float* __restrict__ hist, const Geom g,
                                                              bf16* __restrict__ tab, bf16* __restrict__ planes, int tab_blocks) {
  float v[8];
  bf16* dst;
  size_t pitch;   // from a part to the next
  if ((int)blockIdx.x < tab_blocks) {
    const long long it = (long long)blockIdx.x * 256 + threadIdx.x;
    if (it >= (long long)3 * g.entries * 8 * g.K) return;
    const int k = (int)(it % g.K), r = (int)(it / g.K) & 7;   // neighbouring threads: the filters of one tap row
    const int e = (int)(it / (8 * g.K)) % g.entries, kind = (int)(it / (8ll * g.K * g.entries));
    const int top = 120 - 8 * (e - 16 * (g.nb - 1)) + r;
#pragma unroll
    for (int w = 0; w < 8; w++) {
      const int dist = top - w, j = tap_of(kind, dist);
      v[w] = dist >= 0 && j >= 0 && j < g.L ? phi[(size_t)j * g.K + k] : 0.f;
    }
    dst = tab + (((size_t)(k * 3 + kind) * g.entries + e) * 3 * 8 + r) * 8;
    pitch = 64;
  } else {
    const long long it = (long long)(blockIdx.x - tab_blocks) * 256 + threadIdx.x, per = g.Lp / 8, rows2 = 2ll * g.B * g.d;
    if (it >= rows2 * per) return;
    const long long row = it / per;
    const int s0 = (int)(it - row * per) * 8, n = (g.t_end - (int)(row & 1) + 1) >> 1;
    const float* src = hist + (size_t)row * g.Lh + s0;
#pragma unroll
    for (int w = 0; w < 8; w++) v[w] = s0 + w < n ? src[w] : 0.f;
    dst = planes + (size_t)row * g.Lp + s0;
    pitch = (size_t)rows2 * g.Lp;
  }
  uint4 p[3];
  split2(v[0], v[1], p[0].x, p[1].x, p[2].x);
  split2(v[2], v[3], p[0].y, p[1].y, p[2].y);
  split2(v[4], v[5], p[0].z, p[1].z, p[2].z);
  split2(v[6], v[7], p[0].w, p[1].w, p[2].w);
#pragma unroll
  for (int i = 0; i < 3; i++) *reinterpret_cast<uint4*>(dst + i * pitch) = p[i];
}

__device__ __forceinline__ uint64_t make_desc_sw128(uint32_t saddr) {   // B: K-major, 128-byte swizzle
  return (uint64_t)((saddr >> 4) & 0x3FFF) | (uint64_t)1 << 16 | (uint64_t)(1024 >> 4) << 32 | (uint64_t)1 << 46 | (uint64_t)2 << 61;
}
__device__ __forceinline__ uint64_t make_desc_table(uint32_t saddr) {   // A: core matrices CM bytes apart in either direction
  return (uint64_t)((saddr >> 4) & 0x3FFF) | (uint64_t)(CM >> 4) << 16 | (uint64_t)(CM >> 4) << 32 | (uint64_t)1 << 46;
}
__device__ __forceinline__ void umma(uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(tmem_d), "l"(da), "l"(db), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void umma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(tma::smem_u32(bar))
               : "memory");
}
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,"
      "%28,%29,%30,%31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
        "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
        "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr));
}

struct Tile {
  int mb, ct, p, k;
};
__device__ __forceinline__ Tile tile_at(const Geom& g, int i) {
  Tile t;
  t.k = i % g.K;
  i /= g.K;
  t.p = i & 1;
  i >>= 1;
  t.ct = i % g.n_ct;
  t.mb = g.nb - 1 - i / g.n_ct;
  return t;
}

// A warp's outputs of a tile once more, on the CUDA cores, and stored: lane = position 2 m + p (the warp's 32 m are m_min .. m_min + 31), `half` channels
// from col0 on (16 at a time), filter k.  Entries in steps of AGAIN_S through the warp's staging block; an output meets those that its sum has
// and no others.
constexpr int AGAIN_S = 32, AGAIN_C = 16, AGAIN_TAPS = 32 + AGAIN_S;
static_assert(4 * (2 * AGAIN_S * AGAIN_C + 2 * AGAIN_TAPS) <= STG_BYTES, "staging block");
__device__ __noinline__ void outputs_again(const float* hist, const float* phi, float* U, const Geom& g, int k, int p, int m_min, int m, int col0,
                                           int half, float* st) {
  const int lane = threadIdx.x & 31, rows = g.B * g.d, back = p ? 0 : 1;   // Q: odd taps 2 (m - s - back) + 1
  float *same = st, *other = st + AGAIN_S * AGAIN_C, *te = st + 2 * AGAIN_S * AGAIN_C, *tq = te + AGAIN_TAPS;
  for (; half > 0 && col0 < rows; col0 += AGAIN_C, half -= AGAIN_C) {
    float e[AGAIN_C], q[AGAIN_C];
#pragma unroll
    for (int c = 0; c < AGAIN_C; c++) e[c] = q[c] = 0.f;
    for (int s0 = 0; s0 <= m_min + 31; s0 += AGAIN_S) {
      __syncwarp();
      float v[2][AGAIN_C];   // (all on their way at once)
#pragma unroll
      for (int c = 0; c < AGAIN_C; c++) {
        const int s = s0 + lane;
        const float* h = hist + (size_t)(col0 + c) * 2 * g.Lh + s;
        v[0][c] = col0 + c < rows && 2 * s + p < g.t_end ? h[p ? g.Lh : 0] : 0.f;
        v[1][c] = col0 + c < rows && 2 * s + (p ^ 1) < g.t_end ? h[p ? 0 : g.Lh] : 0.f;
      }
#pragma unroll
      for (int c = 0; c < AGAIN_C; c += 4) {
        *reinterpret_cast<float4*>(same + lane * AGAIN_C + c) = make_float4(v[0][c], v[0][c + 1], v[0][c + 2], v[0][c + 3]);
        *reinterpret_cast<float4*>(other + lane * AGAIN_C + c) = make_float4(v[1][c], v[1][c + 1], v[1][c + 2], v[1][c + 3]);
      }
      const int d0 = m_min - s0 - (AGAIN_S - 1);   // distance that the staged taps begin with
#pragma unroll
      for (int i = lane; i < AGAIN_TAPS; i += 32) {
        const int je = 2 * (d0 + i), jq = 2 * (d0 + i - back) + 1;
        te[i] = je >= 0 && je < g.L ? phi[(size_t)je * g.K + k] : 0.f;
        tq[i] = jq >= 0 && jq < g.L ? phi[(size_t)jq * g.K + k] : 0.f;
      }
      __syncwarp();
      const auto add = [&](float (&sum)[AGAIN_C], float tap, const float* x, int i) {
#pragma unroll
        for (int c = 0; c < AGAIN_C; c += 4) {
          const float4 w = *reinterpret_cast<const float4*>(x + i * AGAIN_C + c);
          sum[c] = fmaf(tap, w.x, sum[c]), sum[c + 1] = fmaf(tap, w.y, sum[c + 1]);
          sum[c + 2] = fmaf(tap, w.z, sum[c + 2]), sum[c + 3] = fmaf(tap, w.w, sum[c + 3]);
        }
      };
      const int at = m - m_min + AGAIN_S - 1;   // tap of entry s0
      if (d0 >= back && 2 * (d0 + AGAIN_TAPS) < g.L) {   // every tap of every lane
#pragma unroll 4
        for (int i = 0; i < AGAIN_S; i++) {
          add(e, te[at - i], same, i);
          add(q, tq[at - i], other, i);
        }
      } else {
#pragma unroll 1
        for (int i = 0; i < AGAIN_S; i++) {
          const int dist = m - s0 - i;
          if (dist >= 0 && 2 * dist < g.L) add(e, te[at - i], same, i);
          if (dist >= back && 2 * (dist - back) + 1 < g.L) add(q, tq[at - i], other, i);
        }
      }
    }
    const int t = 2 * m + p;
    if (t >= g.t0 && t < g.t_end)
#pragma unroll
      for (int c = 0; c < AGAIN_C; c++) {
        const int col = col0 + c, b = col / g.d;
        if (col >= rows) continue;
        float* at = U + ((size_t)b * g.Tn + (t - g.t0)) * g.ldU + (size_t)k * g.d + (col - b * g.d);
        at[0] = e[c] + q[c];
        if (g.both) at[(size_t)g.K * g.d] = e[c] - q[c];
      }
  }
  __syncwarp();
}

template <int TN>
__global__ void __launch_bounds__(THREADS, 1)
    full_conv_f32_umma_kernel(const __grid_constant__ CUtensorMap tmH, const bf16* __restrict__ tab, const float* __restrict__ hist,
                              const float* __restrict__ phi, float* __restrict__ U, const __grid_constant__ Geom g, int* status,
                              int drop_first_stage, unsigned long long wait_ns) {
  constexpr int PLANE_B = plane_b<TN>(), B_PITCH = 3 * PLANE_B, HALF = TN / 2;
  constexpr int A_OFF = STAGES * B_PITCH, STG_OFF = stages_bytes<TN>(), CTL_OFF = STG_OFF + EPI_WARPS * STG_BYTES;
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  Ctl* ctl = reinterpret_cast<Ctl*>(smem + CTL_OFF);
  volatile int* abort_flag = &ctl->abort_flag;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int tiles = (g.nb - g.mb_first) * g.n_ct * 2 * g.K;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; s++) {
      tma::mbar_init(&ctl->full[s], 1);
      tma::mbar_init(&ctl->empty[s], 1);
    }
    for (int i = 0; i < ACCS; i++) {
      tma::mbar_init(&ctl->acc_full[i], 1);
      tma::mbar_init(&ctl->acc_empty[i], EPI_WARPS);
    }
    ctl->abort_flag = 0;
    ctl->issued = ctl->consumed = 0;
    tma::fence_barrier_init();
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(tma::smem_u32(&ctl->tmem_slot)));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::);
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_base = ctl->tmem_slot;

  if (warp == 0) {
    // -------------------------------------------------------------------- producer
    const bool leader = elect_one();
    int it = 0, s = 0;
    uint32_t ph = 1;
    bool ok = true;
    for (int i = blockIdx.x; ok && i < tiles; i += gridDim.x) {
      const Tile t = tile_at(g, i);
      for (int acc = 0; ok && acc < 2; acc++) {   // E, then Q
        const int kind = acc == 0 ? 0 : (t.p ? 1 : 2);
        const bf16* tk = tab + (size_t)(t.k * 3 + kind) * g.entries * (CM / 2);
        for (int kb = 0; kb <= 2 * t.mb + 1; kb++, it++) {
          ok = tma::warp_wait_bounded(&ctl->empty[s], ph, abort_flag, wait_ns);
          if (!ok) break;
          if (leader) tma::mbar_expect_tx(&ctl->full[s], B_PITCH + A_BYTES);
          if (leader && !(drop_first_stage && it == 0)) {   // (a test: these copies are never issued)
            tma::load_4d(smem + s * B_PITCH, &tmH, &ctl->full[s], kb * BK, t.p ^ acc, t.ct * TN, 0);
            const int e0 = 16 * (g.nb - 1) - 16 * t.mb + 8 * kb;   // X = -(m0 - s0) / 8
            tma::bulk_load(smem + A_OFF + s * A_PITCH, tk + (size_t)e0 * (CM / 2), A_BYTES, &ctl->full[s]);
          }
          __syncwarp();
          if (++s == STAGES) s = 0, ph ^= 1u;
        }
      }
    }
    if (leader) ctl->issued = it;
  } else if (warp == 1) {
    // -------------------------------------------------------------------- MMA issuer
    constexpr uint32_t IDESC = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(TN >> 3) << 17) | ((uint32_t)(BM >> 4) << 24);
    const bool leader = elect_one();
    const uint64_t da0 = make_desc_table(tma::smem_u32(smem + A_OFF)), db0 = make_desc_sw128(tma::smem_u32(smem));
    int it = 0, s = 0, a = 0;
    uint32_t ph = 0, aph = 1;
    bool ok = true;
    for (int i = blockIdx.x; ok && i < tiles; i += gridDim.x) {
      const Tile t = tile_at(g, i);
      for (int kb = 0; kb < 2 * (2 * t.mb + 2); kb++, it++) {   // the blocks of E, then those of Q
        ok = tma::warp_wait_bounded(&ctl->full[s], ph, abort_flag, wait_ns);
        if (!ok) break;
        const uint64_t da = da0 + (uint64_t)(s * (A_PITCH >> 4)), db = db0 + (uint64_t)(s * (B_PITCH >> 4));
        ok = tma::warp_wait_bounded(&ctl->acc_empty[a], aph, abort_flag, wait_ns);
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        if (leader) {
#pragma unroll
          for (int p = 0; p < SPLIT_PRODUCTS; p++)
#pragma unroll
            for (int kk = 0; kk < BK / 16; kk++)   // 16 positions: two core matrices of the table, 32 bytes of a history row
              umma(tmem_base + 128 * a, da + (uint64_t)((2 * kk * CM + split_a(p) * 128) >> 4),
                   db + (uint64_t)((split_b(p) * PLANE_B + kk * 32) >> 4), IDESC | split_sign(p), p || kk ? 1u : 0u);
          umma_commit(&ctl->empty[s]);
          umma_commit(&ctl->acc_full[a]);
        }
        __syncwarp();
        if (++a == ACCS) a = 0, aph ^= 1u;
        if (++s == STAGES) s = 0, ph ^= 1u;
      }
    }
    if (leader) ctl->consumed = it;
  } else {
    // -------------------------------------------------------------------- sums and outputs (TMEM lane quarter = warp % 4)
    const int quarter = warp & 3, half = (warp - 2) >> 2;
    float* st = reinterpret_cast<float*>(smem + STG_OFF + (warp - 2) * STG_BYTES);
    const int piece = lane & 7, r0 = lane >> 3;
    const int rows_total = g.B * g.d;
    const uint32_t taddr = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(half * HALF);
    int a = 0;
    uint32_t aph = 0;
    bool ok = true;
    for (int i = blockIdx.x; ok && i < tiles; i += gridDim.x) {
      const Tile t = tile_at(g, i);
      float e[HALF], q[HALF];
#pragma unroll
      for (int c = 0; c < HALF; c++) e[c] = q[c] = 0.f;
      auto add = [&](float (&sum)[HALF]) {
        for (int n = 0; n < 2 * t.mb + 2; n++) {
          if (!tma::warp_wait_bounded(&ctl->acc_full[a], aph, abort_flag, wait_ns)) return false;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
          for (int h = 0; h < HALF; h += 32) {
            uint32_t r[32];
            tmem_ld32(taddr + 128 * a + h, r);
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
            for (int c = 0; c < 32; c++) sum[h + c] += __uint_as_float(r[c]);
          }
          asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
          __syncwarp();
          if (lane == 0) tma::mbar_arrive(&ctl->acc_empty[a]);
          if (++a == ACCS) a = 0, aph ^= 1u;
        }
        return true;
      };
      ok = add(e) && add(q);
      if (!ok) break;
      bool fine = true;
#pragma unroll
      for (int c = 0; c < HALF; c++) {
        e[c] *= SPLIT_UNSCALE, q[c] *= SPLIT_UNSCALE;
        fine = fine && isfinite(e[c]) && isfinite(q[c]);
      }
      if (!__all_sync(0xffffffffu, fine)) {
        // row `lane` of the warp's 32 is position 120 - 8 (L / 8) + L % 8 of the block, L = 32 quarter + lane
        const int m_min = t.mb * BM + 96 - 32 * quarter;
        outputs_again(hist, phi, U, g, t.k, t.p, m_min, m_min + 24 - 8 * (lane >> 3) + (lane & 7), t.ct * TN + half * HALF, HALF, st);
        continue;
      }
#pragma unroll
      for (int sign = 0; sign < 2; sign++) {
        if (sign && !g.both) break;
#pragma unroll
        for (int h = 0; h < HALF; h += 32) {
#pragma unroll
          for (int c = 0; c < 32; c += 4)
            *reinterpret_cast<float4*>(st + lane * SROW + c) =
                sign ? make_float4(e[h + c] - q[h + c], e[h + c + 1] - q[h + c + 1], e[h + c + 2] - q[h + c + 2], e[h + c + 3] - q[h + c + 3])
                     : make_float4(e[h + c] + q[h + c], e[h + c + 1] + q[h + c + 1], e[h + c + 2] + q[h + c + 2], e[h + c + 3] + q[h + c + 3]);
          __syncwarp();
          const int col = t.ct * TN + half * HALF + h + piece * 4;   // four channels of one sequence (d % 4 == 0)
          if (col < rows_total) {
            const int b = col / g.d, c = col - b * g.d;
            float* base = U + (size_t)b * g.Tn * g.ldU + (size_t)(sign * g.K + t.k) * g.d + c;
            float4 v[8];
#pragma unroll
            for (int x = 0; x < 8; x++) v[x] = *reinterpret_cast<const float4*>(st + (r0 + 4 * x) * SROW + piece * 4);
            // row r0 + 4 x of the warp's 32 is position 120 - 8 (L / 8) + L % 8 of the block, L = 32 quarter + r0 + 4 x
            auto time_of = [&](int x) { return 2 * (t.mb * BM + 120 - 32 * quarter - 8 * (x >> 1) + r0 + 4 * (x & 1)) + t.p; };
#pragma unroll
            for (int x = 0; x < 8; x++) {
              const int tt = time_of(x);
              if (tt >= g.t0 && tt < g.t_end) *reinterpret_cast<float4*>(base + (size_t)(tt - g.t0) * g.ldU) = v[x];
            }
          }
          __syncwarp();
        }
      }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  }
  __syncthreads();
  if (*abort_flag) {
    // A wait ran out.  Report it and let the copies that were issued but never consumed land (bounded).
    if (threadIdx.x == 0) {
      if (status) atomicExch(status, STATUS_CONV_WAIT);
      const uint64_t t_start = tma::global_ns();
      for (int it = ctl->consumed; it < ctl->issued; it++)
        for (uint32_t w = 0; w < (1u << 22); ++w) {
          if (tma::mbar_try_wait(&ctl->full[it % STAGES], (uint32_t)(it / STAGES) & 1u)) break;
          if ((w & 255u) == 255u && tma::global_ns() - t_start > wait_ns) break;
        }
    }
    __syncthreads();
  }
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem_base));
  }
}

int blocks_of(int t_end) { return ((t_end + 1) / 2 + BM - 1) / BM; }
int parts_pitch(int t_end) { return ((t_end + 1) / 2 + 7) / 8 * 8; }
long long table_elems(int K, int t_end) { return (long long)K * 3 * table_entries(blocks_of(t_end)) * (CM / 2); }

template <int TN>
int launch_conv(const CUtensorMap& tmH, const bf16* tab, const float* hist, const float* phi, float* U, const Geom& g, int* status,
                cudaStream_t st) {
  static SmemLimit limit;
  const cudaError_t e = allow_smem((const void*)full_conv_f32_umma_kernel<TN>, smem_bytes<TN>(), limit);
  if (e != cudaSuccess) return (int)e;
  const int sms = device_sm_count(), tiles = (g.nb - g.mb_first) * g.n_ct * 2 * g.K;
  full_conv_f32_umma_kernel<TN><<<tiles < sms ? tiles : sms, THREADS, smem_bytes<TN>(), st>>>(tmH, tab, hist, phi, U, g, status, (int)take_dropped_stage(),
                                                                                                            wait_bound_ns());
  STU_CHECK_LAUNCH();
  return STU_OK;
}

}  // namespace

// bf16 elements of scratch of a call that ends at position t_end: the parts of the taps, as operand tables, and of the history.
extern "C" long long stu_full_conv_f32_tc5_scratch_elems(int B, int d, int K, int t_end) {
  if (B <= 0 || d <= 0 || K <= 0 || t_end <= 0) return 0;
  return table_elems(K, t_end) + 6ll * B * d * parts_pitch(t_end);
}

// U[b][t - t0][sign][k][i] (row stride ldU) of positions [t0, t_end) from the history [B][d][2][Lh]; phi [L][K]; all fp32.
// Whether this takes less time than the kernel of stu_full_conv.cu.  Both are waves of tiles: there of 64 entries of both parities and 32 (16) channels, 1.3 us per
// 32 entries where the SMs have three tiles each and 1.6 for one, here of 128 entries of a parity and 128 (64) channels, 1.1 (0.9) us per 64 entries, behind a
// launch that splits the operands.  Fitted to 5461 calls of 1 to 32 sequences, 4 to 1024 channels, 1 to 32 filters and up to 6000 positions: half a percent of
// them are taken and more than 3 % slower (at most 1.26), where the positions alone decided it was a ninth (up to 1.7: 4 x 144 channels of 219 positions, one
// filter, 10.8 us and 15.8).
extern "C" int stu_full_conv_f32_tc5_pays(int B, int d, int K, int t0, int t_end) {
  if (B <= 0 || d <= 0 || K <= 0 || t0 < 0 || t_end <= t0) return 0;
  const long long rows = (long long)B * d, hi = (t_end + 1) / 2, lo = t0 / 2, sms = device_sm_count();
  if (d % 4 || !(t_end >= 400 || (t_end >= 200 && rows >= 512))) return 0;
  const auto up = [](long long a, long long b) { return (a + b - 1) / b; };
  // tensor cores: tiles of the last block come first, the SM with one more than the others has about the mean of first and last
  const bool wide = rows > 64;
  const long long blocks = up(hi, 128), per_block = up(rows, wide ? 128 : 64) * 2 * K, tiles = (blocks - lo / 128) * per_block, waves = up(tiles, sms);
  const long long last = blocks - 1 - (waves - 1) * sms / per_block, stages = waves * (2 * (blocks - 1 + last) + 4);
  const double tensor = 7.15 + stages * (wide ? 1.09 + 0.067 * std::min(tiles, sms) / sms : 0.907) + (wide ? 2.67 * waves : 0.0) +
                        12.5e-6 * (384.0 * blocks * K + rows * hi / 4.0);
  // CUDA cores
  const long long tall = up(hi - lo, 64), columns = K * up(rows, rows <= 16 ? 16 : 32), longest = up(hi, 32);
  const long long steps = columns * ((tall - 1) * up(lo, 32) + tall * (tall - 1) + longest + tall);
  const double cores = 3.5 + std::max(1.6 * longest, (rows <= 16 ? 0.79 : 1.3) * steps / sms + 0.85 * longest);
  return tensor < 0.98 * cores;
}

extern "C" int stu_full_conv_f32_tc5(const void* hist, int Lh, const void* phi, int L, int K, void* scratch, void* U, long long ldU, int B,
                                     int d, int both_signs, int t0, int t_end, int* status, int dtype, void* stream) {
  if (!hist || !phi || !scratch || !U) return STU_ERR_NULL;
  if (B <= 0 || d <= 0 || K <= 0 || L <= 0 || t0 < 0 || t_end <= t0 || t_end > 2 * Lh) return STU_ERR_SHAPE;
  if (dtype != STU_F32) return STU_ERR_DTYPE;
  if (d % 4 || ldU % 4 || !aligned16(scratch) || !aligned16(U)) return STU_ERR_ALIGN;
  if (ldU < (long long)(both_signs ? 2 : 1) * K * d) return STU_ERR_SHAPE;
  const long long rows = (long long)B * d;
  if (rows > (1ll << 30)) return STU_ERR_UNSUPPORTED;
  Geom g;
  g.B = B; g.d = d; g.K = K; g.L = L; g.Lh = Lh; g.Tn = t_end - t0; g.t0 = t0; g.t_end = t_end; g.both = both_signs; g.ldU = ldU;
  g.nb = blocks_of(t_end);
  g.mb_first = (t0 >> 1) / BM;
  g.entries = table_entries(g.nb);
  g.Lp = parts_pitch(t_end);
  const int tn = rows <= 64 ? 64 : 128;
  g.n_ct = (int)((rows + tn - 1) / tn);
  const long long tiles = (long long)(g.nb - g.mb_first) * g.n_ct * 2 * K;
  const long long tab_blocks = ((long long)3 * g.entries * 8 * K + 255) / 256, part_blocks = (2 * rows * (g.Lp / 8) + 255) / 256;
  if (tiles > 0x7fffffffll || tab_blocks + part_blocks > 0x7fffffffll) return STU_ERR_UNSUPPORTED;
  bf16 *tab = (bf16*)scratch, *planes = tab + table_elems(K, t_end);
  CUtensorMap tmH;
  {
    // (position inside the parity, parity, channel row, part)
    cuuint64_t dims[4] = {(cuuint64_t)g.Lp, 2, (cuuint64_t)rows, 3};
    cuuint64_t str[3] = {(cuuint64_t)g.Lp * 2, (cuuint64_t)g.Lp * 4, (cuuint64_t)rows * g.Lp * 4};
    cuuint32_t box[4] = {BK, 1, (cuuint32_t)tn, 3};
    const int rc = tma::encode_bf16(&tmH, planes, 4, dims, str, box, true);
    if (rc != STU_OK) return rc;
  }
  cudaStream_t st = (cudaStream_t)stream;
  full_conv_parts_kernel<<<(unsigned)(tab_blocks + part_blocks), 256, 0, st>>>((const float*)phi, (const float*)hist, g, tab, planes,
                                                                              (int)tab_blocks);
  STU_CHECK_LAUNCH();
  if (tn == 64) return launch_conv<64>(tmH, tab, (const float*)hist, (const float*)phi, (float*)U, g, status, st);
  return launch_conv<128>(tmH, tab, (const float*)hist, (const float*)phi, (float*)U, g, status, st);
}
