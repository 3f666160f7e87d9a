// fp32 GEMM on the 5th-generation tensor cores: y = epilogue(x @ W^T) for fp32 operands, to fp32 accuracy.
//
// Every operand value is split into three bf16 values that add up to it exactly (split3.cuh), and the product is the sum of six of their
// products.  bf16 products are exact in the tensor core; its fp32 sums are not rounded to nearest, so chains of them are kept short:
// an accumulator takes 32 of K, the smallest products first, and is then added to fp32 sums in registers.  Error
// against float64, this kernel and the CUDA-core GEMM (2-norm, normal operands): K = 3072 1.4e-7 and 7.0e-7, 1024 1.2e-7 and 5.7e-7, 256
// 7.7e-8 and 1.5e-7; positive ones (sums that are not rounded to nearest drift) 9.5e-8 and 4.2e-7, 9.4e-8 and 4.3e-7, 6.7e-8 and
// 7.0e-8; 64 of K per accumulator 1.25e-7, 1.1e-7, 8.9e-8, positive 9.7e-8, 9.6e-8, 8.7e-8.  (The weight-streaming kernels of up to 64
// rows are below either and keep those.)
//
// Bound: shared memory, through which a block of 64 of K passes three times as planes and six times as operands, and the splitting, about
// 6 instructions a value.  us, the CUDA-core GEMM and this kernel: 8000 x 96 x 3072 159 and 53, 256 x 512 x 6144 56 and 28, gate/up 256 x 6144 x
// 512 86 and 43, 1000 x 1536 x 512 51 and 23, 4000 x 8192 x 1024 1603 and 487 (138 TFLOP/s of fp32 products, the CUDA cores' peak is 74).
//
// One 128 x BN tile per CTA (gate/up: BN / 2 columns of either), K split over a cluster of KS CTAs whose sums meet in distributed
// shared memory, in rank order.  Warps 0..10 fetch 64 of K of both operands into registers, one block ahead, split them and store the
// three planes in the 128-byte swizzle that the operand descriptors expect, into one of two or three stages; warp 11 issues 24
// tcgen05.mma per block; warps 12..19 drain the accumulators in tensor memory (tcgen05.ld) into their sums.
// Sums that are not finite are computed again on the CUDA cores, 32 rows and half of a tile's columns at a time: operands that are not finite, or
// above 2^87, have no such split, and sums above 2^79 overflow.  4000 x 8192 x 1024, all of them, 6.4 ms (a thread's chain for each, 125 ms; the
// CUDA-core GEMM 1.6), 1000 x 1536 x 512 with a NaN in one row 157 us (36 without).
// Every wait is bounded: on expiry the CTA raises status 3, frees its tensor memory and returns, and no CTA of its cluster stores anything.
#include <cooperative_groups.h>

#include <atomic>

#include "common.cuh"
#include "epilogue.cuh"
#include "split3.cuh"
#include "tma.cuh"

int device_sm_count();      // gemm_tc.cu
int* device_status_word();  // gemm_tc.cu

namespace cg = cooperative_groups;

namespace {

constexpr int BM = 128, BK = 64;
constexpr int CONV_WARPS = 11, ISSUER = 11, DRAIN0 = 12, DRAIN_WARPS = 8, THREADS = 32 * (DRAIN0 + DRAIN_WARPS);
constexpr int CHAIN = 2, CHAINS = BK / 16 / CHAIN;   // steps of 16 of K per accumulator, accumulators per block
constexpr int PLANE_A = BM * BK * 2;

__device__ __forceinline__ uint64_t make_desc(uint32_t saddr) {   // K-major, 128-byte swizzle, 8-row groups 1024 bytes apart
  return (uint64_t)((saddr >> 4) & 0x3FFF) | (uint64_t)1 << 16 | (uint64_t)(1024 >> 4) << 32 | (uint64_t)1 << 46 | (uint64_t)2 << 61;
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
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(tma::smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
        "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
}

struct Ctl {
  uint64_t full[3], empty[3], acc_full[4], acc_empty[4];
  uint32_t tmem_slot;
  int abort_flag;
};

template <int BN> __host__ __device__ constexpr int stage_bytes() { return 3 * (PLANE_A + BN * BK * 2); }
template <int BN> __host__ __device__ constexpr int stages() { return BN <= 64 ? 3 : 2; }
template <int BN> __host__ __device__ constexpr int smem_bytes() { return stages<BN>() * stage_bytes<BN>() + (int)sizeof(Ctl) + 1024; }

// One warp's 32 rows and HALF columns of a tile once more, on the CUDA cores: sums over k in [k0, k1) into part (lane: a row; columns `step` apart).
// room: again_floats() values of shared memory.  Of A there are `rows` rows; B (and B2: gate/up) are those of the tile's columns, of which there are `cols`.
constexpr int AGAIN_K = 32;
template <int HALF> __host__ __device__ constexpr int again_floats() { return 32 * (AGAIN_K + 1) + AGAIN_K * (HALF + 4); }
template <int HALF, int COLS, bool DUAL>
__device__ __noinline__ void sums_again(const float* A, long long lda, int rows, const float* B, const float* B2, long long ldb, int c0, int cols,
                                        int k0, int k1, float* room, float* part, int step) {
  const int lane = threadIdx.x & 31, piece = 4 * (lane & 7);   // 16-byte pieces of a row: K and k0 are multiples of 4 values, rows lie on the grid
  float *a_s = room, *b_s = room + 32 * (AGAIN_K + 1);
  for (int c = 0; c < HALF; c++) part[c * step] = 0.f;
  for (int k = k0; k < k1; k += AGAIN_K) {
    const bool in = k + piece < k1;
    float4 v[8];   // (eight on their way at once)
    __syncwarp();
#pragma unroll
    for (int i = 0; i < 8; i++) {
      const int r = 4 * i + (lane >> 3);
      v[i] = in && r < rows ? *reinterpret_cast<const float4*>(A + (size_t)r * lda + k + piece) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
#pragma unroll
    for (int i = 0; i < 8; i++) {
      float* at = a_s + (4 * i + (lane >> 3)) * (AGAIN_K + 1) + piece;
      at[0] = v[i].x, at[1] = v[i].y, at[2] = v[i].z, at[3] = v[i].w;
    }
#pragma unroll 1
    for (int c8 = 0; c8 < HALF; c8 += 32) {
#pragma unroll
      for (int i = 0; i < (HALF < 32 ? HALF / 4 : 8); i++) {
        const int c = c0 + c8 + 4 * i + (lane >> 3), n = DUAL ? c % COLS : c;
        v[i] = in && n < cols ? *reinterpret_cast<const float4*>((DUAL && c >= COLS ? B2 : B) + (size_t)n * ldb + k + piece) : make_float4(0.f, 0.f, 0.f, 0.f);
      }
#pragma unroll
      for (int i = 0; i < (HALF < 32 ? HALF / 4 : 8); i++) {
        float* at = b_s + piece * (HALF + 4) + c8 + 4 * i + (lane >> 3);
        at[0] = v[i].x, at[HALF + 4] = v[i].y, at[2 * (HALF + 4)] = v[i].z, at[3 * (HALF + 4)] = v[i].w;
      }
    }
    __syncwarp();
#pragma unroll 1
    for (int h = 0; h < HALF; h += 16) {
      float s[16];
#pragma unroll
      for (int c = 0; c < 16; c++) s[c] = 0.f;
#pragma unroll 4
      for (int i = 0; i < AGAIN_K; i++) {
        const float a = a_s[lane * (AGAIN_K + 1) + i];
#pragma unroll
        for (int c = 0; c < 16; c += 4) {
          const float4 b = *reinterpret_cast<const float4*>(b_s + i * (HALF + 4) + h + c);
          s[c] = fmaf(a, b.x, s[c]), s[c + 1] = fmaf(a, b.y, s[c + 1]), s[c + 2] = fmaf(a, b.z, s[c + 2]), s[c + 3] = fmaf(a, b.w, s[c + 3]);
        }
      }
#pragma unroll
      for (int c = 0; c < 16; c++) part[(h + c) * step] += s[c];
    }
  }
}

template <int EPI, int KS, int BN>
__global__ void __launch_bounds__(THREADS, 1)
    gemm_f32_umma_kernel(const float* __restrict__ A, long long lda, const float* __restrict__ B, long long ldb,
                         const float* __restrict__ B2, int M, int N, int K, EpiArgs<float> ep, int* status,
                         int drop_first_stage, unsigned long long wait_ns) {
  constexpr bool DUAL = (EPI == EPI_GELU_MUL), HIST = (EPI == EPI_HIST);
  constexpr int COLS = DUAL ? BN / 2 : BN, STAGE = stage_bytes<BN>(), PLANE_B = BN * BK * 2, PITCH = BN + 4;
  constexpr int STAGES = stages<BN>(), ACCS = BN <= 64 ? 4 : 2, ACC_COLS = BN <= 64 ? 64 : 128;
  constexpr int AT_ONCE = 4 * CONV_WARPS, PIECES = (BM + BN + AT_ONCE - 1) / AT_ONCE;   // rows, 8 threads each; pieces of 8 values per thread
  constexpr int HALF = BN / 2;   // columns of a draining warp
  constexpr uint32_t IDESC = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(BM >> 4) << 24);
  static_assert(BM * PITCH * 4 <= STAGES * STAGE, "the partial tile takes the place of the stages");
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  Ctl* ctl = reinterpret_cast<Ctl*>(smem + STAGES * STAGE);
  // the tile's sums, at the end: rows or, where consecutive threads will take consecutive rows, columns one behind the other
  float* part = reinterpret_cast<float*>(smem);
  const auto at_part = [](int row, int c) { return HIST ? c * BM + row : row * PITCH + c; };
  volatile int* abort_flag = &ctl->abort_flag;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * COLS;
  const int nkb = (K + BK - 1) / BK, per = (nkb + KS - 1) / KS;
  const int kb0 = KS > 1 ? min(nkb, (int)blockIdx.z * per) : 0, kb1 = KS > 1 ? min(nkb, kb0 + per) : nkb;

  if (tid == 0) {
    for (int s = 0; s < STAGES; s++) {
      tma::mbar_init(&ctl->full[s], CONV_WARPS);
      tma::mbar_init(&ctl->empty[s], 1);
    }
    for (int s = 0; s < 4; s++) {
      tma::mbar_init(&ctl->acc_full[s], 1);
      tma::mbar_init(&ctl->acc_empty[s], DRAIN_WARPS);
    }
    ctl->abort_flag = 0;
    tma::fence_barrier_init();
  }
  if (warp == ISSUER) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 256;" ::"r"(tma::smem_u32(&ctl->tmem_slot)));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::);
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_base = ctl->tmem_slot;
  pdl_wait();      // barriers and tensor memory are set up beside the end of the kernel in front
  pdl_trigger();

  const int blocks = kb1 - kb0;
  if (warp < DRAIN0) {
    if (warp < CONV_WARPS) {
      // ---------------- fetch and split; piece i of a thread: values 8 (tid % 8) on of row tid / 8 + 44 i, those of A before those of B
      const int q = tid & 7, r0 = tid >> 3;
      const float* src[PIECES];   // (rows past the last one: that one again, their sums are not stored)
#pragma unroll
      for (int i = 0; i < PIECES; i++) {
        const int r = r0 + AT_ONCE * i, c = min(r - BM, BN - 1);
        src[i] = (r < BM ? A + (size_t)min(m0 + r, M - 1) * lda
                         : (DUAL && c >= COLS ? B2 : B) + (size_t)min(n0 + (DUAL && c >= COLS ? c - COLS : c), N - 1) * ldb) + kb0 * BK + 8 * q;
      }
      float4 v[PIECES][2];
      const int room = K - kb0 * BK - 8 * q;   // values of a row from this thread's first on (K % 4 == 0)
      auto fetch = [&](int i, int n) {
        v[i][0] = n * BK < room ? __ldg(reinterpret_cast<const float4*>(src[i] + n * BK)) : make_float4(0.f, 0.f, 0.f, 0.f);
        v[i][1] = n * BK + 4 < room ? __ldg(reinterpret_cast<const float4*>(src[i] + n * BK + 4)) : make_float4(0.f, 0.f, 0.f, 0.f);
      };
      if (blocks > 0) {
#pragma unroll
        for (int i = 0; i < PIECES; i++) fetch(i, 0);
      }
      int s = 0;
      uint32_t turn = 1;
      for (int n = 0; n < blocks; n++) {
        if (!tma::warp_wait_bounded(&ctl->empty[s], turn, abort_flag, wait_ns)) break;
#pragma unroll
        for (int i = 0; i < PIECES; i++) {
          const int r = r0 + AT_ONCE * i, rr = r < BM ? r : r - BM, plane = r < BM ? PLANE_A : PLANE_B;
          unsigned char* dst = smem + s * STAGE + (r < BM ? 0 : 3 * PLANE_A) + (rr >> 3) * 1024 + (rr & 7) * 128 + ((q ^ (rr & 7)) << 4);
          uint4 w1, w2, w3;
          split2(v[i][0].x, v[i][0].y, w1.x, w2.x, w3.x);
          split2(v[i][0].z, v[i][0].w, w1.y, w2.y, w3.y);
          split2(v[i][1].x, v[i][1].y, w1.z, w2.z, w3.z);
          split2(v[i][1].z, v[i][1].w, w1.w, w2.w, w3.w);
          if (n + 1 < blocks) fetch(i, n + 1);
          if (r < BM + BN) {
            *reinterpret_cast<uint4*>(dst) = w1;
            *reinterpret_cast<uint4*>(dst + plane) = w2;
            *reinterpret_cast<uint4*>(dst + 2 * plane) = w3;
          }
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        // (drop_first_stage, a test: the last CTA of a cluster never has its first block)
        if (lane == 0 && !(drop_first_stage && n == 0 && (KS == 1 || blockIdx.z == KS - 1))) tma::mbar_arrive(&ctl->full[s]);
        if (++s == STAGES) s = 0, turn ^= 1u;
      }
    } else {
      // ---------------- MMA issuer
      const bool leader = elect_one();
      const uint64_t da0 = make_desc(tma::smem_u32(smem)), db0 = make_desc(tma::smem_u32(smem + 3 * PLANE_A));
      int s = 0;
      uint32_t turn = 0;
      for (int n = 0; n < blocks; n++) {
        if (!tma::warp_wait_bounded(&ctl->full[s], turn, abort_flag, wait_ns)) break;
        const uint64_t da = da0 + (uint64_t)(s * (STAGE >> 4)), db = db0 + (uint64_t)(s * (STAGE >> 4));
        bool ok = true;
#pragma unroll
        for (int h = 0; h < CHAINS; h++) {
          const int f = n * CHAINS + h, a = f % ACCS;
          ok = tma::warp_wait_bounded(&ctl->acc_empty[a], ((uint32_t)(f / ACCS) & 1u) ^ 1u, abort_flag, wait_ns);
          if (!ok) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint32_t acc = tmem_base + ACC_COLS * a;
          if (leader) {
#pragma unroll
            for (int p = 0; p < SPLIT_PRODUCTS; p++)
#pragma unroll
              for (int kk = 0; kk < CHAIN; kk++)
                umma(acc, da + ((split_a(p) * PLANE_A + 32 * (h * CHAIN + kk)) >> 4), db + ((split_b(p) * PLANE_B + 32 * (h * CHAIN + kk)) >> 4), IDESC | split_sign(p), p || kk ? 1u : 0u);
            if (h + 1 == CHAINS) umma_commit(&ctl->empty[s]);
            umma_commit(&ctl->acc_full[a]);
          }
          __syncwarp();
        }
        if (!ok) break;
        __syncwarp();
        if (++s == STAGES) s = 0, turn ^= 1u;
      }
    }
    __syncwarp();
    __syncthreads();   // every block has been multiplied: the sums take the place of the stages
  } else {
    // ---------------- drain: TMEM lane quarter = warp % 4, one row per thread, half of the columns
    float sum[HALF];
#pragma unroll
    for (int c = 0; c < HALF; c++) sum[c] = 0.f;
    const int c0 = (warp - DRAIN0) / 4 * HALF;
    const uint32_t at = tmem_base + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)c0;
    for (int n = 0; n < blocks * CHAINS; n++) {
      const int a = n % ACCS;
      if (!tma::warp_wait_bounded(&ctl->acc_full[a], (uint32_t)(n / ACCS) & 1u, abort_flag, wait_ns)) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
      for (int h = 0; h < HALF; h += 16) {
        uint32_t r[16];
        tmem_ld16(at + ACC_COLS * a + h, r);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
        for (int c = 0; c < 16; c++) sum[h + c] += __uint_as_float(r[c]);
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) tma::mbar_arrive(&ctl->acc_empty[a]);
    }
    __syncwarp();
    __syncthreads();
    const int r0 = (warp & 3) * 32;
    float* p = part + at_part(r0 + lane, c0);
    bool fine = true;
#pragma unroll
    for (int c = 0; c < HALF; c++) {
      sum[c] *= SPLIT_UNSCALE;
      fine = fine && isfinite(sum[c]);
      if (HIST) p[c * BM] = sum[c];
    }
#pragma unroll
    for (int c = 0; c < (HIST ? 0 : HALF); c += 4) *reinterpret_cast<float4*>(p + c) = make_float4(sum[c], sum[c + 1], sum[c + 2], sum[c + 3]);
    if (!__all_sync(0xffffffffu, fine)) {
      constexpr int ROOM = (BM * PITCH + 31) / 32 * 32;   // behind the tile's sums
      static_assert(4 * (ROOM + DRAIN_WARPS * again_floats<HALF>()) <= STAGES * STAGE, "room for the sums made again");
      sums_again<HALF, COLS, DUAL>(A + (size_t)min(m0 + r0, M - 1) * lda, lda, min(32, M - m0 - r0), B + (size_t)n0 * ldb, DUAL ? B2 + (size_t)n0 * ldb : nullptr, ldb, c0,
                                   N - n0, kb0 * BK, min(kb1 * BK, K), part + ROOM + (warp - DRAIN0) * again_floats<HALF>(), p, HIST ? BM : 1);
    }
  }
  cg::cluster_group cluster = cg::this_cluster();
  if (KS > 1 && tid == 0 && *abort_flag) {   // nobody adds up sums that one of the cluster has not got
    if (status) atomicExch(status, 3);
    for (int r = 0; r < KS; r++) *cluster.map_shared_rank(&ctl->abort_flag, r) = 1;
  }
  if constexpr (KS > 1) cluster.sync(); else __syncthreads();
  const int rank = KS > 1 ? (int)cluster.block_rank() : 0;
  const float* parts[KS];
#pragma unroll
  for (int r = 0; r < KS; r++) parts[r] = KS > 1 ? cluster.map_shared_rank(part, r) : part;
  if (!*abort_flag) {
    // This CTA's outputs are the tile's rows rank, rank + KS, ...; of a history, which is time-major, its columns rank, rank + KS, ..., whose sums lie one
    // behind the other (in rows, four to 32 lanes met in a bank: 114 x 2912 x 292 29 us, now 11).  Residuals are read four at a time (4944 x 3891 x 96
    // 190 -> 124 us), over a cluster singly: a CTA has few of them, and with four (or two) the compiler's main loop is 6 % slower (388 x 256 x 12288 53.3, now 49.9).
    constexpr int OUTS = BM / KS * COLS, AT_A_TIME = EPI == EPI_RESID && KS > 1 ? 1 : 4;
    const auto output = [&](int e, int& m, int& n, float& s, float& s2) {
      const int row = HIST ? e % BM : rank + e / COLS * KS, c = HIST ? rank + e / BM * KS : e % COLS;
      m = m0 + row, n = n0 + c, s = s2 = 0.f;
      if (e >= OUTS || m >= M || n >= N) return false;
#pragma unroll
      for (int r = 0; r < KS; r++) {
        s += parts[r][at_part(row, c)];
        if (DUAL) s2 += parts[r][at_part(row, COLS + c)];
      }
      return true;
    };
    for (int e0 = tid; e0 < OUTS; e0 += AT_A_TIME * THREADS) {
      float s[AT_A_TIME], s2[AT_A_TIME], r[AT_A_TIME];
      int m[AT_A_TIME], n[AT_A_TIME];
      bool in[AT_A_TIME];
#pragma unroll
      for (int i = 0; i < AT_A_TIME; i++) {
        in[i] = output(e0 + i * THREADS, m[i], n[i], s[i], s2[i]);
        r[i] = EPI == EPI_RESID && in[i] ? ep.resid[(size_t)m[i] * ep.ldr + n[i]] : 0.f;   // (all ahead of the stores, which they might alias)
      }
#pragma unroll
      for (int i = 0; i < AT_A_TIME; i++) {
        if (!in[i]) continue;
        if (EPI == EPI_RESID) ep.y[(size_t)m[i] * ep.ldy + n[i]] = r[i] + s[i];
        else epilogue_store<float, EPI>(ep, m[i], n[i], s[i], s2[i]);
      }
    }
  } else if (tid == 0 && status) {
    atomicExch(status, 3);
  }
  if constexpr (KS > 1) cluster.sync(); else __syncthreads();   // the other CTAs' sums stay alive until read
  if (warp == ISSUER) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 256;" ::"r"(tmem_base));
  }
}

struct Operands {
  const float *A, *B, *B2;
  long long lda, ldb;
  int M, N, K;
};

// How many clusters of KS CTAs the GPU holds at a time (the SMs of a GPC are no multiple of 8: 8 leave some of them out); 0: none, or it cannot say now
template <int EPI, int KS, int BN>
int clusters_at_once() {
  static std::atomic<int> known[STU_MAX_DEVICES] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= STU_MAX_DEVICES) dev = 0;
  int n = KS == 1 ? device_sm_count() : known[dev].load(std::memory_order_relaxed);
  if (n != 0) return n < 0 ? 0 : n;
  auto kern = gemm_f32_umma_kernel<EPI, KS, BN>;
  static SmemLimit limit;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(1, 1, KS);
  cfg.blockDim = dim3(THREADS);
  cfg.dynamicSmemBytes = smem_bytes<BN>();
  cudaLaunchAttribute at;
  at.id = cudaLaunchAttributeClusterDimension;
  at.val.clusterDim.x = at.val.clusterDim.y = 1;
  at.val.clusterDim.z = KS;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  if (allow_smem((const void*)kern, smem_bytes<BN>(), limit) != cudaSuccess || cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess) {
    (void)cudaGetLastError();   // (asked again by the next call)
    return 0;
  }
  known[dev].store(n > 0 ? n : -1, std::memory_order_relaxed);
  return n;
}
template <int EPI, int BN>
int clusters_at_once(int ks) {
  return ks == 1 ? clusters_at_once<EPI, 1, BN>() : ks == 2 ? clusters_at_once<EPI, 2, BN>() : ks == 4 ? clusters_at_once<EPI, 4, BN>() : clusters_at_once<EPI, 8, BN>();
}

template <int EPI, int KS, int BN>
int launch_tile(const Operands& o, const EpiArgs<float>& ep, cudaStream_t st) {
  constexpr int COLS = EPI == EPI_GELU_MUL ? BN / 2 : BN;
  auto kern = gemm_f32_umma_kernel<EPI, KS, BN>;
  static SmemLimit limit;
  cudaError_t e = allow_smem((const void*)kern, smem_bytes<BN>(), limit);
  if (e != cudaSuccess) return (int)e;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((o.N + COLS - 1) / COLS, (o.M + BM - 1) / BM, KS);
  cfg.blockDim = dim3(THREADS);
  cfg.dynamicSmemBytes = smem_bytes<BN>();
  cfg.stream = st;
  cudaLaunchAttribute at[2];
  int n = 0;
  if (pdl_enabled()) {
    at[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[n++].val.programmaticStreamSerializationAllowed = 1;
  }
  if (KS > 1) {
    at[n].id = cudaLaunchAttributeClusterDimension;
    at[n].val.clusterDim.x = 1;
    at[n].val.clusterDim.y = 1;
    at[n++].val.clusterDim.z = KS;
  }
  cfg.attrs = at;
  cfg.numAttrs = n;
  e = cudaLaunchKernelEx(&cfg, kern, o.A, o.lda, o.B, o.ldb, o.B2, o.M, o.N, o.K, ep, device_status_word(), (int)take_dropped_stage(), wait_bound_ns());
  if (e != cudaSuccess) return (int)e;
  STU_CHECK_LAUNCH();
  return STU_OK;
}

template <int EPI, int BN>
int launch_split(const Operands& o, int ks, const EpiArgs<float>& ep, cudaStream_t st) {
  switch (ks) {
    case 1: return launch_tile<EPI, 1, BN>(o, ep, st);
    case 2: return launch_tile<EPI, 2, BN>(o, ep, st);
    case 4: return launch_tile<EPI, 4, BN>(o, ep, st);
    default: return launch_tile<EPI, 8, BN>(o, ep, st);
  }
}

// The tile width and the split of K that take the least time: waves of clusters, a CTA per SM, of 4.2 us and 1.05, 1.5 or 1.95 us per block of
// 64 of K (32, 64 or 128 columns), 0.8 us and a tenth per CTA of a cluster (fitted to 26 shapes of 20 to 8192 rows; within 10 % of the best of
// all in each).  clusters(columns, ks): how many the GPU holds at a time; a split of which it holds none is not taken, and of single CTAs it holds some.
template <typename Clusters>
void choose_tile(int M, int N, int K, bool dual, const Clusters& clusters, int* best_bn, int* best_ks) {
  const int blocks = (K + BK - 1) / BK;
  double best = 1e30;
  *best_bn = 128, *best_ks = 1;
  for (int bn = 128; bn >= 32; bn /= 2)
    for (int ks = 1; ks <= 8 && (ks == 1 || blocks >= ks); ks *= 2) {
      const int cols = dual ? bn / 2 : bn, room = clusters(bn, ks);
      if (room < 1) continue;
      const long long tiles = (long long)((M + BM - 1) / BM) * ((N + cols - 1) / cols);
      const double block = bn == 128 ? 1.95 : bn == 64 ? 1.5 : 1.05;
      const double t = (double)((tiles + room - 1) / room) * (4.2 + (blocks + ks - 1) / ks * block + (ks > 1 ? 0.8 + 0.1 * ks : 0.0));
      if (t < best) best = t, *best_bn = bn, *best_ks = ks;
    }
}

template <int EPI>
int launch_epi(const Operands& o, const EpiArgs<float>& ep, cudaStream_t st) {
  int best_bn, best_ks;
  choose_tile(o.M, o.N, o.K, EPI == EPI_GELU_MUL, [](int bn, int ks) {
    return bn == 128 ? clusters_at_once<EPI, 128>(ks) : bn == 64 ? clusters_at_once<EPI, 64>(ks) : clusters_at_once<EPI, 32>(ks);
  }, &best_bn, &best_ks);
  switch (best_bn) {
    case 32: return launch_split<EPI, 32>(o, best_ks, ep, st);
    case 64: return launch_split<EPI, 64>(o, best_ks, ep, st);
    default: return launch_split<EPI, 128>(o, best_ks, ep, st);
  }
}

}  // namespace

// Test hook: columns * 16 + CTAs per cluster of the tiles of a product on a GPU that holds room[i] clusters of 2^i CTAs at a time.
extern "C" int stu_test_f32_tile(int M, int N, int K, int gate_up, const int* room) {
  int bn, ks;
  choose_tile(M, N, K, gate_up != 0, [room](int, int of) { return room[of == 1 ? 0 : of == 2 ? 1 : of == 4 ? 2 : 3]; }, &bn, &ks);
  return bn * 16 + ks;
}

// Both operands K-major with rows on the 16-byte grid; from 256 of K on, or from 96 where the tiles of 64 x 64 are four per SM and more (us, the
// CUDA-core GEMM and this one: 4000 x 4096 x 64 62 and 64, x 96 87 and 74; 8000 x 96 x 96 9.2 and 10.9; 300 x 512 x 128 7.8 and 8.4).  Where
// the CUDA-core GEMM splits K into eight chains of less than 128 it is as fast and, for positive operands, a tenth more exact.  Lower-triangular weights stay there: their
// short rows are such sums, and it reads nothing past blocks of 64 columns (what lies there need not be finite).
bool gemm_f32_umma_takes(const void* A, long long lda, const void* B, long long ldb, long long skb, const void* B2, int M, int N, int K,
                         int causal, int dtype) {
  if (causal || dtype != STU_F32 || skb != 1 || lda % 4 || ldb % 4 || K % 4 || !aligned16(A) || !aligned16(B) || (B2 && !aligned16(B2))) return false;
  if (M <= 64 || N < 1) return false;
  const long long tiles = (long long)((M + 63) / 64) * ((N + 63) / 64), sms = device_sm_count();
  if (K < 256) return K >= 96 && tiles >= 4 * sms;
  return K >= 1024 || tiles * 4 >= 2 * sms;
}

int gemm_f32_umma_dispatch(const void* A, long long lda, const void* B, long long ldb, const void* B2, int M, int N, int K, int epi,
                           const EpiArgsAny& ep, cudaStream_t st) {
  const Operands o{(const float*)A, (const float*)B, (const float*)B2, lda, ldb, M, N, K};
  switch (epi) {
    case EPI_STORE: return launch_epi<EPI_STORE>(o, ep.as<float>(), st);
    case EPI_RESID: return launch_epi<EPI_RESID>(o, ep.as<float>(), st);
    case EPI_GELU_MUL: return launch_epi<EPI_GELU_MUL>(o, ep.as<float>(), st);
    case EPI_HIST: return launch_epi<EPI_HIST>(o, ep.as<float>(), st);
    case EPI_BLOCKCOL: return launch_epi<EPI_BLOCKCOL>(o, ep.as<float>(), st);
  }
  return STU_ERR_UNSUPPORTED;
}
