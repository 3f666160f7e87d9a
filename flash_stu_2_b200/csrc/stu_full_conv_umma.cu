// Prefill convolutions of the full STU variant on the 5th-generation tensor cores, all filters in one launch
// (flash_stu/modules/stu.py:100-118; MiniSTU mini_stu/stu.py:240-269).
//
//   U+-[b,t,k,i] = sum_j (+-1)^j phi[j,k] x[b,t-j,i]
//
// With the history parity-split (hist[b][i][p][s], time t = 2 s + p) the even and the odd taps give, per filter k,
//   E[m, (b,i,p)] = sum_{s<=m} phi[2(m-s), k] hist[b,i,p][s],      Q[m, (b,i,p)] = sum_s phi[2(m-s)+-1, k] hist[b,i,1-p][s]
// and U+- = E +- Q, rounded to bf16 as E and Q are.  A tile is 128 positions m x up to 256 channels of one parity and one
// filter: E and Q are two products with lower-triangular Toeplitz matrices (the A operand: rows are positions, so that the
// result leaves in token rows) and the same history rows (the B operand, K-major as they lie).
//
// No Toeplitz matrix is materialised: in the un-swizzled K-major operand layout a 128 x 64 block is a grid of 8 x 8
// core matrices, and with the row groups in descending order core matrix (q', kc) depends on q' + kc alone.  A table of
// core matrices CM[X][r][w] = f[dist + 120 - 8 X + r - w] per filter and tap set (26 KB for 3000 positions) therefore holds
// every block, and a stage of 64 columns brings 23 consecutive entries of it (3 KB) where a block would be 16 KB.
//
// Bound: the tensor pipe (2 * 2 S^2/2 multiply-adds per channel pair and filter) beside the 2 K d values written per
// token.  E stays in registers, as the bf16 values it is rounded to, while Q is accumulated in the other half of tensor
// memory; so neither goes through memory.  One filter at a time with materialised matrices, E and Q in memory and a kernel
// to combine them, 24 filters over 8 sequences of 3000 x 1024 took 121 launches and 3.4 ms; this form 2 launches and 1.6 ms (the
// layer's prefill and 64 steps: 10.25 -> 8.42 ms, the same values).
//
// Roles (one persistent CTA per SM, 320 threads): warp 0 producer, warp 1 MMA issuer, warps 2-9 epilogue (a quarter of the
// rows and every other 64-channel block each).  Tiles run from the latest positions (the most work) down, the filters of
// a channel block side by side, so that its history rows are read from L2.  Every load is a plain single-CTA copy of this
// GPU's own memory.  Every wait is bounded: on expiry the CTA raises status 9, lets issued copies land (bounded), frees its
// tensor memory and returns.
#include <cuda.h>

#include "common.cuh"
#include "tma.cuh"

int device_sm_count();

namespace {

constexpr int BM = 128, BK = 64;
constexpr int A_ENTRIES = 23;                  // core matrices of a 128 x 64 block: q' + kc = 0 .. 15 + 7
constexpr int A_BYTES = A_ENTRIES * 128;
constexpr int A_PITCH = 3072;
constexpr int B_BYTES = 256 * BK * 2;
constexpr int STAGES = 5;
constexpr int SROW = 72;                       // row distance of the epilogue's staging block (as in the GEMM)
constexpr int A_OFF = STAGES * B_BYTES;
constexpr int STG_OFF = A_OFF + STAGES * A_PITCH;
constexpr int STG_BYTES = 32 * SROW * 2;       // per warp
constexpr int EPI_WARPS = 8;
constexpr int CTL_OFF = STG_OFF + EPI_WARPS * STG_BYTES;
constexpr int SMEM_BYTES = CTL_OFF + 256 + 1024;
constexpr int THREADS = 64 + 32 * EPI_WARPS;
constexpr int STATUS_CONV_WAIT = 9;

struct Ctl {
  uint64_t full[STAGES], empty[STAGES], acc_full[2], acc_empty[2];
  uint32_t tmem_slot;
  int abort_flag, issued, consumed;
};
static_assert(sizeof(Ctl) <= 256, "control block");
static_assert(SMEM_BYTES <= 227 * 1024, "shared memory");

struct Geom {
  int B, d, K, Tn, t0, t_end;
  int both;               // U- too
  int tn;                 // channels per tile: 64, 128 or 256
  int mb_first, nb;       // 128-position blocks with outputs: mb_first .. nb - 1
  int n_ct;               // channel tiles
  int entries;            // table entries per filter and tap set
  long long ldU;
};

// Tap sets: 0 even taps, 1 odd taps of outputs of parity 1 from inputs of parity 0, 2 odd taps the other way round.
__device__ __forceinline__ int tap_of(int kind, int dist) { return 2 * dist + (kind == 0 ? 0 : (kind == 1 ? 1 : -1)); }
__host__ __device__ inline int table_entries(int nb) { return 16 * (nb - 1) + 31; }

// CM[k][kind][e][r][w]: the tap at distance 120 - 8 X + r - w, X = e - 16 (nb - 1); zero above the diagonal and past
// the filter.  One thread per row (16 bytes).
__global__ void __launch_bounds__(256) full_conv_table_kernel(const bf16* __restrict__ phi, int K, int L, int nb,
                                                              bf16* __restrict__ tab) {
  const int entries = table_entries(nb);
  const int kind = blockIdx.y, total = entries * 8 * K;
  for (int it = blockIdx.x * 256 + threadIdx.x; it < total; it += gridDim.x * 256) {
    const int k = it % K, r = (it / K) & 7, e = it / (8 * K);   // neighbouring threads: the filters of one tap row
    const int top = 120 - 8 * (e - 16 * (nb - 1)) + r;
    bf16 v[8];
#pragma unroll
    for (int w = 0; w < 8; w++) {
      const int dist = top - w, j = tap_of(kind, dist);
      v[w] = dist >= 0 && j >= 0 && j < L ? phi[(size_t)j * K + k] : __float2bfloat16_rn(0.f);
    }
    *reinterpret_cast<uint4*>(tab + (((size_t)(k * 3 + kind) * entries + e) * 8 + r) * 8) = *reinterpret_cast<const uint4*>(v);
  }
}

__device__ __forceinline__ uint64_t make_desc_sw128(uint32_t saddr) {   // B: K-major, 128-byte swizzle
  uint64_t d = 0;
  d |= (uint64_t)((saddr >> 4) & 0x3FFF);
  d |= (uint64_t)1 << 16;
  d |= (uint64_t)(1024 >> 4) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)2 << 61;
  return d;
}
__device__ __forceinline__ uint64_t make_desc_table(uint32_t saddr) {   // A: core matrices 128 bytes apart in either direction
  uint64_t d = 0;
  d |= (uint64_t)((saddr >> 4) & 0x3FFF);
  d |= (uint64_t)(128 >> 4) << 16;
  d |= (uint64_t)(128 >> 4) << 32;
  d |= (uint64_t)1 << 46;
  return d;
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
__device__ __forceinline__ uint32_t pack2(float lo, float hi) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&h);
}
__device__ __forceinline__ float lo_f(uint32_t v) { return __uint_as_float(v << 16); }
__device__ __forceinline__ float hi_f(uint32_t v) { return __uint_as_float(v & 0xffff0000u); }

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

__global__ void __launch_bounds__(THREADS, 1) full_conv_umma_kernel(const __grid_constant__ CUtensorMap tmH,
                                                                    const bf16* __restrict__ tab, bf16* __restrict__ U,
                                                                    const Geom g, int* status, unsigned long long wait_ns) {
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
    for (int i = 0; i < 2; i++) {
      tma::mbar_init(&ctl->acc_full[i], 1);
      tma::mbar_init(&ctl->acc_empty[i], 32 * EPI_WARPS);
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
    const uint32_t bytes = (uint32_t)g.tn * BK * 2 + A_BYTES;
    int it = 0, s = 0;
    uint32_t ph = 1;
    bool ok = true;
    for (int i = blockIdx.x; ok && i < tiles; i += gridDim.x) {
      const Tile t = tile_at(g, i);
      for (int acc = 0; ok && acc < 2; acc++) {   // E, then Q
        const int kind = acc == 0 ? 0 : (t.p ? 1 : 2);
        const bf16* tk = tab + (size_t)(t.k * 3 + kind) * g.entries * 64;
        for (int kb = 0; kb <= 2 * t.mb + 1; kb++, it++) {
          ok = tma::warp_wait_bounded(&ctl->empty[s], ph, abort_flag, wait_ns);
          if (!ok) break;
          if (leader) {
            tma::mbar_expect_tx(&ctl->full[s], bytes);
            tma::load_3d(smem + s * B_BYTES, &tmH, &ctl->full[s], kb * BK, t.p ^ acc, t.ct * g.tn);
            const int e0 = 16 * (g.nb - 1) - 16 * t.mb + 8 * kb;   // X = -(m0 - s0) / 8
            tma::bulk_load(smem + A_OFF + s * A_PITCH, tk + (size_t)e0 * 64, A_BYTES, &ctl->full[s]);
          }
          __syncwarp();
          if (++s == STAGES) s = 0, ph ^= 1u;
        }
      }
    }
    if (leader) ctl->issued = it;
  } else if (warp == 1) {
    // -------------------------------------------------------------------- MMA issuer
    const bool leader = elect_one();
    const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(g.tn >> 3) << 17) | ((uint32_t)(BM >> 4) << 24);
    int it = 0, n = 0, s = 0;
    uint32_t ph = 0;
    bool ok = true;
    for (int i = blockIdx.x; ok && i < tiles; i += gridDim.x, n++) {
      const Tile t = tile_at(g, i);
      for (int acc = 0; ok && acc < 2; acc++) {
        ok = tma::warp_wait_bounded(&ctl->acc_empty[acc], ((uint32_t)n & 1u) ^ 1u, abort_flag, wait_ns);
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        for (int kb = 0; kb <= 2 * t.mb + 1; kb++, it++) {
          ok = tma::warp_wait_bounded(&ctl->full[s], ph, abort_flag, wait_ns);
          if (!ok) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint64_t da = make_desc_table(tma::smem_u32(smem + A_OFF + s * A_PITCH));
          const uint64_t db = make_desc_sw128(tma::smem_u32(smem + s * B_BYTES));
          if (leader) {
#pragma unroll
            for (int kk = 0; kk < BK / 16; kk++)   // 16 columns: two core matrices of the table, 32 bytes of a history row
              umma(tmem_base + acc * 256, da + (uint64_t)(kk * 256 >> 4), db + (uint64_t)(kk * 32 >> 4), idesc, (kb | kk) ? 1u : 0u);
            umma_commit(&ctl->empty[s]);
          }
          __syncwarp();
          if (++s == STAGES) s = 0, ph ^= 1u;
        }
        if (ok && leader) umma_commit(&ctl->acc_full[acc]);
        __syncwarp();
      }
    }
    if (leader) ctl->consumed = it;
  } else {
    // -------------------------------------------------------------------- epilogue (TMEM lane quarter = warp % 4)
    const int quarter = warp & 3, half = (warp - 2) >> 2;
    bf16* st = reinterpret_cast<bf16*>(smem + STG_OFF + (warp - 2) * STG_BYTES);
    const int piece = lane & 7, r0 = lane >> 3;
    const int rows_total = g.B * g.d, nblk = g.tn >> 6;
    int n = 0;
    for (int i = blockIdx.x; i < tiles; i += gridDim.x, n++) {
      const Tile t = tile_at(g, i);
      const uint32_t taddr = tmem_base + ((uint32_t)(quarter * 32) << 16);
      uint32_t e[2][32];   // E of this lane's position, 64 channels each, rounded
      bool ok = tma::mbar_wait_bounded(&ctl->acc_full[0], (uint32_t)n & 1u, abort_flag, wait_ns);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
      for (int j = 0; j < 2; j++) {
        const int blk = half + 2 * j;
        if (blk < nblk) {
#pragma unroll
          for (int h = 0; h < 2; h++) {
            uint32_t r[32];
            tmem_ld32(taddr + blk * 64 + h * 32, r);
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
            for (int x = 0; x < 16; x++) e[j][h * 16 + x] = pack2(__uint_as_float(r[2 * x]), __uint_as_float(r[2 * x + 1]));
          }
        }
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      tma::mbar_arrive(&ctl->acc_empty[0]);
      ok = tma::mbar_wait_bounded(&ctl->acc_full[1], (uint32_t)n & 1u, abort_flag, wait_ns);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      // the warp's 32 positions: lane L of the tile is position 120 - 8 (L / 8) + L % 8
      auto flush = [&](int blk, int sign) {   // the staged 32 x 64 block, 8 lanes per token row
        const int col = t.ct * g.tn + blk * 64 + piece * 8;
        if (col >= rows_total) return;
        const int b = col / g.d, c = col - b * g.d;
        bf16* base = U + (size_t)b * g.Tn * g.ldU + (size_t)(sign * g.K + t.k) * g.d + c;
#pragma unroll
        for (int x = 0; x < 8; x++) {
          const int row = r0 + 4 * x, L = quarter * 32 + row;
          const int tt = 2 * (t.mb * BM + 120 - 8 * (L >> 3) + (L & 7)) + t.p;
          if (tt >= g.t0 && tt < g.t_end)
            *reinterpret_cast<uint4*>(base + (size_t)(tt - g.t0) * g.ldU) = *reinterpret_cast<const uint4*>(st + row * SROW + piece * 8);
        }
      };
#pragma unroll
      for (int j = 0; j < 2; j++) {
        const int blk = half + 2 * j;
        if (blk < nblk) {
#pragma unroll
          for (int h = 0; h < 2; h++) {
            uint32_t r[32];
            tmem_ld32(taddr + 256 + blk * 64 + h * 32, r);
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
            for (int v = 0; v < 4; v++) {
              uint32_t up[4];
#pragma unroll
              for (int x = 0; x < 4; x++) {
                const int y = v * 4 + x;
                const uint32_t q = pack2(__uint_as_float(r[2 * y]), __uint_as_float(r[2 * y + 1])), ev = e[j][h * 16 + y];
                up[x] = pack2(lo_f(ev) + lo_f(q), hi_f(ev) + hi_f(q));
                e[j][h * 16 + y] = pack2(lo_f(ev) - lo_f(q), hi_f(ev) - hi_f(q));
              }
              *reinterpret_cast<uint4*>(st + lane * SROW + h * 32 + v * 8) = make_uint4(up[0], up[1], up[2], up[3]);
            }
          }
          __syncwarp();
          flush(blk, 0);
          __syncwarp();
          if (g.both) {
#pragma unroll
            for (int v = 0; v < 8; v++)
              *reinterpret_cast<uint4*>(st + lane * SROW + v * 8) =
                  make_uint4(e[j][v * 4], e[j][v * 4 + 1], e[j][v * 4 + 2], e[j][v * 4 + 3]);
            __syncwarp();
            flush(blk, 1);
            __syncwarp();
          }
        }
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      tma::mbar_arrive(&ctl->acc_empty[1]);
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

}  // namespace

// bf16 elements of scratch for the core-matrix tables of a call that ends at position t_end.
extern "C" long long stu_full_conv_tc5_scratch_elems(int K, int t_end) {
  if (K <= 0 || t_end <= 0) return 0;
  return (long long)K * 3 * table_entries(blocks_of(t_end)) * 64;
}

// U[b][t - t0][sign][k][i] (row stride ldU) of positions [t0, t_end) from the history [B][d][2][Lh]; phi [L][K].
extern "C" int stu_full_conv_tc5(const void* hist, int Lh, const void* phi, int L, int K, void* scratch, void* U, long long ldU,
                                 int B, int d, int both_signs, int t0, int t_end, int* status, int dtype, void* stream) {
  if (!hist || !phi || !scratch || !U) return STU_ERR_NULL;
  if (B <= 0 || d <= 0 || K <= 0 || L <= 0 || t0 < 0 || t_end <= t0 || t_end > 2 * Lh) return STU_ERR_SHAPE;
  if (dtype != STU_BF16) return STU_ERR_DTYPE;
  if (d % 8 || Lh % 8 || ldU % 8 || !aligned16(hist) || !aligned16(scratch) || !aligned16(U)) return STU_ERR_ALIGN;
  if (ldU < (long long)(both_signs ? 2 : 1) * K * d) return STU_ERR_SHAPE;
  const long long rows = (long long)B * d;
  if (rows > (1ll << 30)) return STU_ERR_UNSUPPORTED;
  Geom g;
  g.B = B; g.d = d; g.K = K; g.Tn = t_end - t0; g.t0 = t0; g.t_end = t_end; g.both = both_signs; g.ldU = ldU;
  g.nb = blocks_of(t_end);
  g.mb_first = (t0 >> 1) / BM;
  g.entries = table_entries(g.nb);
  const int sms = device_sm_count();
  // The widest tile that the rows fill more than half of: a narrower one reads its table block for fewer channels, which shows even
  // where wide ones leave SMs idle.  us, tiles of 64, 128 and 256 channels, 24 filters: 1 x 512 of 100 positions 12.8, 11.5 and
  // 11.4, of 700 33.6, 24.2 and 21.0; 4 x 1024 of 1500 626, 362 and 286; 8 x 1024 of 3000 4159, 2395 and 1886.
  g.tn = 256;
  while (g.tn > 64 && rows <= g.tn / 2) g.tn /= 2;
  g.n_ct = (int)((rows + g.tn - 1) / g.tn);
  const long long tiles = (long long)(g.nb - g.mb_first) * g.n_ct * 2 * K;
  if (tiles > 0x7fffffffll || (long long)g.entries * 8 * K > 0x7fffffffll) return STU_ERR_UNSUPPORTED;
  CUtensorMap tmH;
  {
    // (position inside the parity, parity, channel row); past the last position of the call zeros are read
    cuuint64_t dims[3] = {(cuuint64_t)((t_end + 1) / 2), 2, (cuuint64_t)rows};
    cuuint64_t str[2] = {(cuuint64_t)Lh * 2, (cuuint64_t)Lh * 4};
    cuuint32_t box[3] = {BK, 1, (cuuint32_t)g.tn};
    const int rc = tma::encode_bf16(&tmH, hist, 3, dims, str, box, true);
    if (rc != STU_OK) return rc;
  }
  static SmemLimit limit;
  const cudaError_t e = allow_smem((const void*)full_conv_umma_kernel, SMEM_BYTES, limit);
  if (e != cudaSuccess) return (int)e;
  cudaStream_t st = (cudaStream_t)stream;
  const int rows_tab = g.entries * 8 * K;
  full_conv_table_kernel<<<dim3((rows_tab + 255) / 256, 3), 256, 0, st>>>((const bf16*)phi, K, L, g.nb, (bf16*)scratch);
  STU_CHECK_LAUNCH();
  full_conv_umma_kernel<<<(int)(tiles < sms ? tiles : sms), THREADS, SMEM_BYTES, st>>>(tmH, (const bf16*)scratch, (bf16*)U, g,
                                                                                       status, 2000000000ull);
  STU_CHECK_LAUNCH();
  return STU_OK;
}
