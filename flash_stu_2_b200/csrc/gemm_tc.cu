// Prefill linear layers on the 5th-generation tensor cores: D[M,N] = A[M,K] . B[N,K]^T in bf16 with
// fp32 accumulators held in tensor memory (TMEM).
//
// A pair of CTAs on neighbouring SMs computes 256 x 128 or 256 x 256 output tiles (gate/up: 256 x 128 of both accumulators) with
// tcgen05.mma.cta_group::2: either CTA holds 128 rows of A, half the rows of B and the accumulator of its 128 rows.  What bounds
// the large products is shared memory and power: a CTA alone on a 128 x 256 tile passes 96 KB through shared memory per 64 of K,
// in a pair 64.  Warp 0 of either CTA is its TMA producer (cp.async.bulk.tensor, 128-byte swizzled tiles into a ring of stages,
// counted on the first CTA's barriers), warp 1 allocates TMEM and, in the first CTA, issues the pair's tcgen05.mma; warps 2..9
// drain the accumulator with tcgen05.ld and run the fused epilogue (store / residual add / tanh-GELU gate * up / transposed
// scatter into the projected history).  The kernel is persistent (one pair per two SMs walks the tile list) and the accumulator is
// double-buffered in TMEM, so one tile's epilogue overlaps the next tile's main loop.  Every load is a plain load of this GPU's
// own memory into the loading CTA's shared memory.  Where tiles of 256 rows would fill their last wave badly, CTAs alone on tiles of
// 128 x 256 take their place (tile_form); where long K keeps few of them busy, it is cut (split_plan).
// One CTA per 128 x 256 or 128 x 128 tile, as it was before, and now (us, all back to back): 65536 x 1536 x 6144 938 -> 880,
// gate/up 65536 x 6144 x 1536 1998 -> 1874, 65536 x 4608 x 1536 771 -> 656, 7996 x 3072 x 1024 47.3 -> 43.0, 1668 x 768 x 3072
// 18.1 -> 12.0, 333 x 1536 x 6144 32.0 -> 18.3; smallest 4.3 -> 4.7 (256 x 256 x 64), before the launch became programmatic: barriers and tensor memory
// are set up beside the end of the kernel in front (three turns of 834 positions through 12 layers of 768: 3917 -> 3618 us).
//
// Every wait on an mbarrier is bounded: on expiry the waiter tells the other CTA and raises the status word, the pair drains
// its outstanding bulk copies (bounded as well), frees its TMEM and returns.
#include <cooperative_groups.h>
#include <cuda.h>
#include <stdlib.h>

#include <algorithm>

#include "common.cuh"
#include "epilogue.cuh"

int device_sm_count();   // SM count of the current device (cached per device)
static int current_device();
extern thread_local int t_linear_launches;   // api.cu: kernels of this thread's last linear

namespace cg = cooperative_groups;

namespace {

constexpr int BM = 128, BK = 64;
constexpr int A_BYTES = BM * BK * 2;
constexpr int EPI_WARPS = 8;               // of the prefill kernel
constexpr int BLOCK_BYTES = 32 * 64 * 2;   // an epilogue warp's block of 32 rows x 64 columns in shared memory
constexpr uint32_t WAIT_LIMIT = 1u << 22;
enum { EPI_HIST_T = 4 };  // internal: rows = channels, columns = tokens (operands swapped by the host)

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// Whether the phase is complete, without waiting for it.
__device__ __forceinline__ bool mbar_ready(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// Bounded wait: gives up after WAIT_LIMIT polls or wait_ns of wall time (two seconds unless a test shortened it),
// whichever comes first.
// Returns false when the limit ran out or another role already gave up.
__device__ __forceinline__ uint64_t global_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, volatile int* abort_flag,
                                          unsigned long long wait_ns) {
  uint64_t start = 0;
  for (uint32_t it = 0; it < WAIT_LIMIT; ++it) {
    if (mbar_try_wait(bar, parity)) return true;
    if ((it & 255u) == 255u) {
      if (*abort_flag) return false;
      uint64_t now = global_ns();
      if (start == 0) start = now;
      else if (now - start > wait_ns) break;
    }
  }
  *abort_flag = 1;
  return false;
}

// The same for a whole warp: one answer for all lanes.
__device__ __forceinline__ bool warp_wait(uint64_t* bar, uint32_t parity, volatile int* abort_flag, unsigned long long wait_ns) {
  return __all_sync(0xffffffffu, mbar_wait(bar, parity, abort_flag, wait_ns));
}
__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map, uint64_t* bar, int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(smem_u32(dst)), "l"(map), "r"(smem_u32(bar)), "r"(x), "r"(y)
      : "memory");
}

// The same issued by either CTA of a pair: the tile lands in this CTA's shared memory, the bytes are counted on a barrier of
// the pair's first CTA (`bar`: its shared::cluster address).
__device__ __forceinline__ void tma_load_2d_pair(void* dst, const CUtensorMap* map, uint32_t bar, int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(smem_u32(dst)), "l"(map), "r"(bar), "r"(x), "r"(y)
      : "memory");
}
// shared::cluster address of the pair's first CTA's copy of a shared-memory object
__device__ __forceinline__ uint32_t in_first_cta(const void* p) {
  uint32_t a;
  asm("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(a) : "r"(smem_u32(p)));
  return a;
}
__device__ __forceinline__ uint32_t load_from_cta(const volatile int* p, uint32_t cta) {
  uint32_t a, v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_u32((const void*)p)), "r"(cta));
  asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ void store_to_cta(const volatile int* p, uint32_t cta, int v) {
  uint32_t a;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_u32((const void*)p)), "r"(cta));
  asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}
// Both CTAs of the pair, all threads.  Orders no stores (that would wait for the outputs to arrive): barriers are made visible
// by their own fence, the flag of a CTA that gave up by one ahead of this.
__device__ __forceinline__ void pair_sync() {
  asm volatile("barrier.cluster.arrive.relaxed.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// Shared-memory matrix descriptor for a K-major bf16 tile stored as rows of 128 bytes with the
// 128-byte swizzle (what the tensor maps below produce): 8-row groups are 1024 bytes apart.
__device__ __forceinline__ uint64_t make_smem_desc(uint32_t saddr) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr >> 4) & 0x3FFF);
  d |= (uint64_t)1 << 16;                 // leading byte offset (unused for swizzled K-major), encoded >> 4
  d |= (uint64_t)(1024 >> 4) << 32;       // stride byte offset between 8-row groups
  d |= (uint64_t)1 << 46;                 // descriptor version for this architecture
  d |= (uint64_t)2 << 61;                 // 128-byte swizzle
  return d;
}
// Instruction descriptor: D fp32, A/B bf16, both K-major, M = 128, N = 256 (tiles of single CTAs) or the 16, 32 or 64 rows of a token step.
template <int BN_>
__device__ __forceinline__ void umma(uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t accumulate) {
  constexpr uint32_t IDESC =
      (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BN_ >> 3) << 17) | ((uint32_t)(BM >> 4) << 24);
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(tmem_d), "l"(da), "l"(db), "r"(IDESC), "r"(accumulate)
      : "memory");
}
// One instruction of a CTA pair: M = 256 (128 rows of A from each CTA's shared memory), the N rows of B half in either's.
template <int BN_>
__device__ __forceinline__ void umma_pair(uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t accumulate) {
  constexpr uint32_t IDESC =
      (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BN_ >> 3) << 17) | ((uint32_t)(2 * BM >> 4) << 24);
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(tmem_d), "l"(da), "l"(db), "r"(IDESC), "r"(accumulate)
      : "memory");
}
// Arrives at the barrier of both CTAs when the pair's instructions so far are done.
__device__ __forceinline__ void umma_commit_pair(uint64_t* bar) {
  asm volatile(
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(smem_u32(bar)),
      "h"((uint16_t)3)
      : "memory");
}
__device__ __forceinline__ void umma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
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
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t* r) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr));
}
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const float* v) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};"
               ::"r"(taddr), "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7])
               : "memory");
}

// A barrier of this pair (shared::cluster address).  At the default scope: a release for the cluster waits for all of the
// thread's stores so far to arrive, which nothing here needs (the reads of tensor memory are done and fenced).
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
// tanh-GELU with the hardware tanh approximation (relative error ~2^-11, below the bf16 rounding that follows)
__device__ __forceinline__ float gelu_tanh_fast(float x) {
  const float inner = 0.7978845608028654f * (x + 0.044715f * x * x * x);
  float t;
  asm("tanh.approx.f32 %0, %1;" : "=f"(t) : "f"(inner));
  return 0.5f * x * (1.0f + t);
}

// Two values rounded to bf16 and back: one conversion for both (the conversions bound the gate/up epilogue: 5250 -> 3300 cycles
// of a tile).
__device__ __forceinline__ void round_pair(float& a, float& b) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  const uint32_t w = *reinterpret_cast<const uint32_t*>(&h);
  a = __uint_as_float(w << 16);
  b = __uint_as_float(w & 0xffff0000u);
}
// o = round(gelu(round(o))) * round(up), eight of them
__device__ __forceinline__ void gelu_mul(float* o, const uint32_t* up) {
#pragma unroll
  for (int j = 0; j < 8; j += 2) {
    float u0 = __uint_as_float(up[j]), u1 = __uint_as_float(up[j + 1]);
    round_pair(o[j], o[j + 1]);
    round_pair(u0, u1);
    o[j] = gelu_tanh_fast(o[j]);
    o[j + 1] = gelu_tanh_fast(o[j + 1]);
    round_pair(o[j], o[j + 1]);
    o[j] *= u0;
    o[j + 1] *= u1;
  }
}

// With `causal` the B operand is lower triangular (B[n][k] = 0 for k > n, the Toeplitz matrices of the STU
// full variant): k-blocks that lie entirely above the diagonal of the tile's last column are skipped.
__device__ __forceinline__ int tile_kb(int num_kb, int n0, int causal, int bn) {
  if (!causal) return num_kb;
  const int need = (n0 + bn + BK - 1) / BK;
  return need < num_kb ? need : num_kb;
}

// Column blocks with ep.Lh > 0 (EPI_FLAG_TOEPLITZ): row m of A is zero from column K - Lh + m / t0 + 1 on (the Toeplitz part of the distilled-LDS features,
// t0 rows per position): the k-blocks behind the last row's are skipped (6144 x 48128 x 320, half of whose rows need 256: 184 -> 174 us).
template <int EPI>
__device__ __forceinline__ int row_kb(int kb, const EpiArgs<bf16>& ep, int last_row, int K) {
  if (EPI != EPI_BLOCKCOL || ep.Lh <= 0) return kb;
  return min(kb, (K - ep.Lh + last_row / ep.t0 + BK) / BK);
}

// Tile order: bands of group_m row tiles, rows first inside a band (group_m = 1: row by row; tiles_m: column by
// column).  The host picks group_m, see gemm_group_m.
__device__ __forceinline__ void tile_coords(int tile, int tiles_m, int tiles_n, int group_m, int& tm, int& tn) {
  const int band = tile / (group_m * tiles_n);
  const int r = tile - band * group_m * tiles_n;
  const int rows = min(group_m, tiles_m - band * group_m);
  tn = r / rows;
  tm = band * group_m + (r - tn * rows);
}

// k-blocks per stage of the ring.  Waiting for a stage, issuing and committing cost about 400 cycles whatever the size of the
// instructions: more than the 256 that the four of a 128-column block take, less than the 512 of a 256-column one.  So the narrow
// tiles take two blocks per stage (1536 x 6144 outputs' 333 rows 21.2 -> 18.9 us), the wide ones one, in twice as many stages
// (gate/up of 65536 x 1536 1810 -> 1738 us).
__host__ __device__ constexpr int stage_blocks(int mma_n) { return mma_n > 128 ? 1 : 2; }

// Persistent kernel: pair i of CTAs handles tiles i, i + pairs, ...  The accumulator is double-buffered in TMEM
// (2 x TN columns, or 2 x 256 for the two accumulators of the gate/up epilogue), so the MMA warp starts the next
// tile while the epilogue warps drain the previous one.
// CTAS = 1: the same with a CTA in the place of a pair, tiles of 128 rows (cta_group::1, all rows of B in its shared memory), for
// products whose tiles of 256 rows would fill their last wave badly (see tile_form).
// SPLIT: K of the tiles behind the first `whole` is cut into `parts` (split_plan); what a pair works on are then those tiles' parts, and their
// sums go to `partials` in fp32: per part [CTA][32 rows][4 columns], every store of a warp 512 bytes in a row.  split_sum_kernel adds them up.
// The first `whole` tiles' sums are made of the same parts, one accumulator behind the other and added up in the epilogue's registers in the same order:
// equal rows of x give equal results wherever they stand.
struct SplitK {
  int whole, parts;
  float* partials;
};
constexpr int SPLIT_TILE = 256 * 256;   // values of a part
template <int EPI, int STAGES, int TN, int CTAS, bool SPLIT>
__global__ void __cluster_dims__(CTAS, 1, 1) __launch_bounds__(64 + 32 * EPI_WARPS, 1)
    gemm_tc_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                   const __grid_constant__ CUtensorMap tmB2, const __grid_constant__ CUtensorMap tmY, int by_copy, int M, int N,
                   int K, int tiles_m, int tiles_n, int group_m, int causal, EpiArgs<bf16> ep, int* status,
                   int drop_first_copy, unsigned long long wait_ns, SplitK split) {
  constexpr bool DUAL = (EPI == EPI_GELU_MUL);
  constexpr bool COPIES = (EPI == EPI_STORE || EPI == EPI_GELU_MUL || EPI == EPI_BLOCKCOL);   // outputs that nothing is added to
  constexpr int BN = TN;                       // output columns of a tile
  constexpr int MMA_N = DUAL ? 2 * BN : BN;    // accumulator columns
  constexpr int KBS = stage_blocks(MMA_N);
  constexpr bool PAIR = CTAS == 2;
  constexpr int KB_BYTES = A_BYTES + MMA_N / CTAS * BK * 2;   // of one CTA: its rows of A, its half of B (or all of it)
  constexpr int STAGE_BYTES = KBS * KB_BYTES;
  constexpr uint32_t ACC_COLS = MMA_N;
  constexpr uint32_t TMEM_COLS = MMA_N > 128 ? 512 : 256;     // two accumulators, a power of two
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + STAGES * STAGE_BYTES);   // used in the pair's first CTA alone
  uint64_t* empty_bar = full_bar + STAGES;
  uint64_t* tmem_full = empty_bar + STAGES;   // [2]
  uint64_t* tmem_empty = tmem_full + 2;       // [2], first CTA alone
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tmem_empty + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);   // [2]: this CTA gave up, the other one did
  int* issued_ctr = const_cast<int*>(reinterpret_cast<volatile int*>(tmem_slot + 3));
  int* consumed_ctr = issued_ctr + 1;
  unsigned char* blocks = smem + STAGES * STAGE_BYTES + 1024;   // one per epilogue warp, in the 128-byte swizzle

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = PAIR ? blockIdx.x & 1 : 0, pair = blockIdx.x / CTAS, pairs = gridDim.x / CTAS;
  const int num_tiles = SPLIT ? split.whole + (tiles_m * tiles_n - split.whole) * split.parts : tiles_m * tiles_n;
  int num_kb = (K + BK - 1) / BK;
  // tile and k-blocks of a part.  All tiles' first parts come first: what works on them at a time shares its k-blocks in L2.
  const int rest = SPLIT ? tiles_m * tiles_n - split.whole : 1;
  const auto whole_tile = [&](int tile) { return SPLIT && tile >= split.whole ? split.whole + (tile - split.whole) % rest : tile; };
  const auto part_range = [&](int part, int& kb0, int& kb_end) {
    kb0 = (int)((long long)num_kb * part / split.parts);
    kb_end = (int)((long long)num_kb * (part + 1) / split.parts);
  };
  const auto chains = [&](int tile) { return SPLIT && tile < split.whole ? split.parts : 1; };   // accumulators of a tile
  const auto k_range = [&](int tile, int& kb0, int& kb_end) {
    if (SPLIT && tile >= split.whole) {
      const int part = (tile - split.whole) / rest;
      part_range(part, kb0, kb_end);
    }
  };

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; s++) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int i = 0; i < 2; i++) {
      mbar_init(&tmem_full[i], 1);
      mbar_init(&tmem_empty[i], CTAS * EPI_WARPS);   // of both CTAs
    }
    abort_flag[0] = abort_flag[1] = 0;
    *issued_ctr = 0;
    *consumed_ctr = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    if constexpr (PAIR) {
      asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(TMEM_COLS));
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::);
    } else {
      asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(TMEM_COLS));
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::);
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if constexpr (PAIR) pair_sync();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_base = *tmem_slot;
  // launched programmatically: everything so far ran beside the end of the kernel in front; the next kernel may be made resident
  // once that one is complete (see PdlTrigger, epilogue.cuh) and this one holds its tensor memory
  pdl_wait();
  pdl_trigger();
  if (EPI == EPI_STORE && ep.kpos) num_kb = min(num_kb, max(__ldg(ep.kpos), 0) / (2 * BK) + 1);   // the rest of W is zero

  if (warp == 0) {
    // ---------------- TMA producer (of either CTA: its 128 rows of A, its half of the rows of B)
    const bool leader = elect_one();
    const CUtensorMap* mapB = DUAL && rank ? &tmB2 : &tmB;   // gate/up: the first CTA brings the gate rows, the second the up rows
    const uint32_t full0 = in_first_cta(full_bar);
    int g = 0, s = 0;  // stages issued so far, ring position
    uint32_t ph = 1;
    bool ok = true, ready = false;
    for (int tile = pair; ok && tile < num_tiles; tile += pairs) {
      int tm, tn;
      tile_coords(whole_tile(tile), tiles_m, tiles_n, group_m, tm, tn);
      const int m0 = (CTAS * tm + rank) * BM, n0 = tn * BN + (DUAL ? 0 : rank * (BN / 2));
      int kb0 = 0, kb_end = row_kb<EPI>(tile_kb(num_kb, tn * BN, causal, BN), ep, min((tm + 1) * CTAS * BM, M) - 1, K);
      k_range(tile, kb0, kb_end);
      for (int kb = kb0; kb < kb_end; kb += KBS, g++) {
        if (!ready) ok = warp_wait(&empty_bar[s], ph, abort_flag, wait_ns);
        if (!ok) break;
        const int s1 = s + 1 == STAGES ? 0 : s + 1;
        const uint32_t ph1 = s1 ? ph : ph ^ 1u;
        const bool ready1 = mbar_ready(&empty_bar[s1], ph1);   // asked for here, looked at behind the copies
        if (leader) {
          const int n = min(KBS, kb_end - kb);
          unsigned char* sa = smem + s * STAGE_BYTES;
          if (rank == 0) mbar_expect_tx(&full_bar[s], CTAS * n * KB_BYTES);   // of both CTAs
          // drop_first_copy (failure-detection test only): the first stage's copies are never issued, so its
          // barrier never completes and the consumer's bounded wait has to run out
          if (!(drop_first_copy && g == 0)) {
            const uint32_t bar = full0 + s * (uint32_t)sizeof(uint64_t);
#pragma unroll
            for (int j = 0; j < KBS; j++)
              if (j < n) {
                unsigned char* sj = sa + j * KB_BYTES;
                if constexpr (PAIR) {
                  tma_load_2d_pair(sj, &tmA, bar, (kb + j) * BK, m0);
                  tma_load_2d_pair(sj + A_BYTES, mapB, bar, (kb + j) * BK, n0);
                } else {
                  tma_load_2d(sj, &tmA, &full_bar[s], (kb + j) * BK, m0);
                  tma_load_2d(sj + A_BYTES, &tmB, &full_bar[s], (kb + j) * BK, n0);
                  if (DUAL) tma_load_2d(sj + A_BYTES + BN * BK * 2, &tmB2, &full_bar[s], (kb + j) * BK, n0);   // gate rows, up rows
                }
              }
          }
        }
        ready = __all_sync(0xffffffffu, ready1);
        s = s1, ph = ph1;
      }
    }
    if (leader) *issued_ctr = g;
    // the last stages' releases arrive in both CTAs: wait for them here, so that none is under way to a CTA that has left
    for (int h = max(g - STAGES, 0); ok && h < g; h++)
      ok = warp_wait(&empty_bar[h % STAGES], (uint32_t)(h / STAGES) & 1u, abort_flag, wait_ns);
  } else if (warp == 1) {
    if (rank == 0) {
      // ---------------- MMA issuer of the pair
      const bool leader = elect_one();
      const uint64_t da0 = make_smem_desc(smem_u32(smem)), db0 = make_smem_desc(smem_u32(smem) + A_BYTES);
      int g = 0, s = 0, it = 0;
      uint32_t ph = 0;
      bool ok = true, ready = false;
      for (int tile = pair, chain = 0; ok && tile < num_tiles; it++) {
        const int buf = it & 1;
        const uint32_t acc_addr = tmem_base + (uint32_t)buf * ACC_COLS;
        int tm, tn;
        tile_coords(whole_tile(tile), tiles_m, tiles_n, group_m, tm, tn);
        int kb0 = 0, kb_end = row_kb<EPI>(tile_kb(num_kb, tn * BN, causal, BN), ep, min((tm + 1) * CTAS * BM, M) - 1, K);
        if (chains(tile) > 1) part_range(chain, kb0, kb_end);
        else k_range(tile, kb0, kb_end);
        if (++chain >= chains(tile)) tile += pairs, chain = 0;   // (of the next turn)
        ok = warp_wait(&tmem_empty[buf], (((uint32_t)it >> 1) & 1u) ^ 1u, abort_flag, wait_ns);
        if (!ok) break;
        for (int kb = kb0; kb < kb_end; kb += KBS, g++) {
          if (!ready) ok = warp_wait(&full_bar[s], ph, abort_flag, wait_ns);
          if (!ok) break;
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const int s1 = s + 1 == STAGES ? 0 : s + 1;
          const uint32_t ph1 = s1 ? ph : ph ^ 1u;
          const bool ready1 = mbar_ready(&full_bar[s1], ph1);   // asked for here, looked at behind the instructions
          if (leader) {
            const uint64_t da = da0 + (uint64_t)(s * (STAGE_BYTES >> 4)), db = db0 + (uint64_t)(s * (STAGE_BYTES >> 4));
            // advancing 16 bf16 = 32 bytes along K inside the swizzled row: +2 in the (>>4) address field
            // gate/up: the B operand is the gate tile (first CTA) and the up tile (second), one N = 256 instruction fills
            // both accumulators (columns 0..127 gate, 128..255 up)
#pragma unroll
            for (int j = 0; j < KBS; j++)
              if (j == 0 || kb + j < kb_end) {
#pragma unroll
                for (int kk = 0; kk < BK / 16; kk++) {
                  const uint64_t dak = da + j * (KB_BYTES >> 4) + 2 * kk, dbk = db + j * (KB_BYTES >> 4) + 2 * kk;
                  if constexpr (PAIR) umma_pair<MMA_N>(acc_addr, dak, dbk, ((kb - kb0) | j | kk) ? 1u : 0u);
                  else umma<MMA_N>(acc_addr, dak, dbk, ((kb - kb0) | j | kk) ? 1u : 0u);
                }
              }
            // arrives when the MMAs above have finished reading this stage
            if constexpr (PAIR) umma_commit_pair(&empty_bar[s]);
            else umma_commit(&empty_bar[s]);
          }
          ready = __all_sync(0xffffffffu, ready1);
          s = s1, ph = ph1;
        }
        if (ok && leader) {
          if constexpr (PAIR) umma_commit_pair(&tmem_full[buf]);
          else umma_commit(&tmem_full[buf]);
        }
        __syncwarp();
      }
      if (leader) *consumed_ctr = g;
    }
  } else {
    // ---------------- epilogue warps: TMEM lane quarter = warp % 4
    const int quarter = warp & 3;
    // The accumulator leaves in blocks of 32 rows x 64 columns per warp, through shared memory: a thread holds a row, but
    // 16-byte stores by 32 threads to 32 rows cost 32 half-used sectors per instruction (4.6 us per 128 x 256 tile, more
    // than its main loop below K = 768); 8 threads per row write whole lines (LDS features, 6144 x 48128 x 320: 281 -> 236 us;
    // residual GEMMs of 7996 x 1024: 58 -> 48 us).  Residual rows are read the same way, all
    // eight loads ahead of the first use.  Histories (rows are channels, columns tokens): the even and the odd tokens of a
    // block are 32 values each in their parity rows.
    // Off the 16-byte grid (plain rows of any stride; histories whose sequences, first position or pitch are no multiples
    // of the blocks) lanes store single values, side by side.
    const bool unaligned = EPI == EPI_STORE ? ((ep.ldy & 7) || (reinterpret_cast<uintptr_t>(ep.y) & 15))
                                            : EPI == EPI_HIST_T && ((ep.Tseq & 15) || (ep.t0 & 15) || (ep.Lh & 7));
    // Plain rows off that grid go in shifted pieces (below) unless a main loop that is long enough hides the single stores, which then cost less:
    // from K = 832 on and with more than six tiles per pair.  us, pieces and single values: 1668 x 50257 (18 tiles per pair), K = 768 / 832 / 960 /
    // 1024 / 2048 116 / 134 / 139 / 150 / 251 and 123 / 137 / 133 / 140 / 248; 400 x 50257 (5), K = 1024 54.4 and 54.4; 1668 x 5001 (2), K = 1024 / 2048 18.2 / 27.5 and
    // 19.2 / 28.4; 256 x 32003 (2), K = 1024 / 3072 24.7 / 55.8 and 25.7 / 57.1.
    const bool in_pieces = EPI == EPI_STORE && unaligned && (K <= 832 || num_tiles <= 6 * pairs);
    // Plain outputs leave by tensor copies where they can: one lane sends the block off, edges clipped by the copy, which runs
    // beside the next block's accumulator reads.
    // Eight warps, two per quarter of the rows and either at every other 64 columns: four took 7400 cycles for a gate/up tile
    // and 3900 for 256 columns, more than the main loop of K = 768 (6200) and all of it behind the last tile's.
    bf16* st = reinterpret_cast<bf16*>(blocks + (warp - 2) * BLOCK_BYTES);
    const int half = (warp - 2) >> 2;
    auto at = [&](int row, int piece) { return st + row * 64 + ((piece ^ (row & 7)) << 3); };   // 8 values, 16 bytes
    const uint32_t hand_back = in_first_cta(tmem_empty);
    int it = 0;
    for (int tile = pair; tile < num_tiles; tile += pairs, it++) {
      int tm, tn;
      tile_coords(whole_tile(tile), tiles_m, tiles_n, group_m, tm, tn);
      const int m0 = (CTAS * tm + rank) * BM, n0 = tn * BN;
      const int first = m0 + quarter * 32, rows = min(32, M - first);   // this warp's rows
      bool ok = true;
      if constexpr (SPLIT) {
        if (tile < split.whole) {   // this warp's part of the tile, 32 rows and 64 of every 128 columns, over all accumulators but the last, and that one's on top
          float sum[128];
#pragma unroll
          for (int i = 0; i < 128; i++) sum[i] = -0.f;   // (the zero that leaves the sign of another alone)
          for (int chain = 0;; chain++, it++) {
            ok = mbar_wait(&tmem_full[it & 1], ((uint32_t)it >> 1) & 1u, abort_flag, wait_ns);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t taddr = tmem_base + (uint32_t)(it & 1) * ACC_COLS + ((uint32_t)(quarter * 32) << 16) + 64 * half;
#pragma unroll
            for (int i = 0; i < 16; i++) {
              uint32_t r[8];
              tmem_ld8(taddr + (i >> 3) * 128 + (i & 7) * 8, r);
              asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
              for (int j = 0; j < 8; j++) sum[8 * i + j] += __uint_as_float(r[j]);
            }
            if (chain + 1 == split.parts) {
#pragma unroll
              for (int i = 0; i < 16; i++) tmem_st8(taddr + (i >> 3) * 128 + (i & 7) * 8, sum + 8 * i);
              break;
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(hand_back + (it & 1) * (uint32_t)sizeof(uint64_t));
          }
          if (!ok) break;
          asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");   // read again below, by this warp
        }
      }
      const int buf = it & 1;
      const uint32_t acc_addr = tmem_base + (uint32_t)buf * ACC_COLS;
      if (!SPLIT || tile >= split.whole) {
        ok = mbar_wait(&tmem_full[buf], ((uint32_t)it >> 1) & 1u, abort_flag, wait_ns);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      }
      if (SPLIT && tile >= split.whole) {
        float4* part = reinterpret_cast<float4*>(split.partials + (size_t)(tile - split.whole) * SPLIT_TILE) + (rank * 4 + quarter) * (BN / 4) * 32 + lane;
#pragma unroll 1
        for (int nb = n0 + 64 * half; nb < (rows > 0 ? min(n0 + BN, N) : 0); nb += 128) {
          const uint32_t taddr = acc_addr + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(nb - n0);
          uint32_t r[2][32];
          tmem_ld32(taddr, r[0]);
          tmem_ld32(taddr + 32, r[1]);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
          for (int j = 0; j < 16; j++)
            part[((nb - n0) / 4 + j) * 32] = make_float4(__uint_as_float(r[j >> 3][4 * (j & 7)]), __uint_as_float(r[j >> 3][4 * (j & 7) + 1]),
                                                         __uint_as_float(r[j >> 3][4 * (j & 7) + 2]), __uint_as_float(r[j >> 3][4 * (j & 7) + 3]));
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(hand_back + buf * (uint32_t)sizeof(uint64_t));
        continue;
      }
      if (COPIES && by_copy) {
#pragma unroll 1
        for (int nb = n0 + 64 * half; nb < min(n0 + BN, N); nb += 128) {
          const uint32_t taddr = acc_addr + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(nb - n0);
#pragma unroll
          for (int h = 0; h < 2; h++) {
            uint32_t r[32], r2[32];
            tmem_ld32(taddr + h * 32, r);
            if (DUAL) tmem_ld32(taddr + BN + h * 32, r2);
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
            if (h == 0) {
              if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");   // the block before has left
              __syncwarp();
            }
#pragma unroll
            for (int v8 = 0; v8 < 4; v8++) {
              float o[8];
#pragma unroll
              for (int j = 0; j < 8; j++) o[j] = __uint_as_float(r[v8 * 8 + j]);
              if (DUAL) gelu_mul(o, r2 + v8 * 8);
              store_vec(at(lane, h * 4 + v8), o);
            }
          }
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
          __syncwarp();
          if (lane == 0) {
            if (rows <= 0) {
            } else if (EPI == EPI_BLOCKCOL)
              asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.bulk_group [%0, {%2, %3, %4}], [%1];" ::"l"(&tmY),
                           "r"(smem_u32(st)), "r"(nb % ep.Tseq), "r"(first), "r"(nb / ep.Tseq)
                           : "memory");
            else
              asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];" ::"l"(&tmY),
                           "r"(smem_u32(st)), "r"(nb), "r"(first)
                           : "memory");
            asm volatile("cp.async.bulk.commit_group;" ::: "memory");
          }
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(hand_back + buf * (uint32_t)sizeof(uint64_t));
        continue;
      }
#pragma unroll 1
      for (int nb = n0 + 64 * half; nb < min(n0 + BN, N); nb += 128) {
        const uint32_t taddr = acc_addr + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(nb - n0);
        const bool shifted = in_pieces && nb + 64 <= N;
#pragma unroll 1
        for (int h = 0; h < 2; h++) {   // 32 columns of this thread's row
          uint32_t r[32], r2[32];
          tmem_ld32(taddr + h * 32, r);
          if (DUAL) tmem_ld32(taddr + BN + h * 32, r2);
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
          if (EPI == EPI_HIST_T && !unaligned) {
            float par[2][16];
#pragma unroll
            for (int j = 0; j < 32; j++) par[j & 1][j >> 1] = __uint_as_float(r[j]);
#pragma unroll
            for (int q = 0; q < 2; q++) {
              store_vec(at(lane, q * 4 + h * 2), par[q]);
              store_vec(at(lane, q * 4 + h * 2 + 1), par[q] + 8);
            }
          } else {
#pragma unroll
            for (int v8 = 0; v8 < 4; v8++) {
              float o[8];
#pragma unroll
              for (int j = 0; j < 8; j++) o[j] = __uint_as_float(r[v8 * 8 + j]);
              if (DUAL) gelu_mul(o, r2 + v8 * 8);
              store_vec(at(lane, h * 4 + v8), o);
            }
          }
          if (unaligned && !shifted) {   // 32 columns at a time: the stores of one half run beside the accumulator read of the next
            __syncwarp();
            const int n = nb + h * 32 + lane;
            if (n < N) {
              const int piece = h * 4 + (lane >> 3), c = lane & 7;
              if (EPI == EPI_HIST_T) {
                const int b = n / ep.Tseq, pitch = 2 * ep.Lh;
                bf16* yc = ep.y + hist_off(b, first, ep.t0 + (n - b * ep.Tseq), (int)ep.ldy, ep.Lh);
#pragma unroll 8
                for (int i = 0; i < rows; i++) yc[(size_t)i * pitch] = at(i, piece)[c];
              } else {
                bf16* yc = ep.y + (size_t)first * ep.ldy + n;
#pragma unroll 8
                for (int i = 0; i < rows; i++) yc[(size_t)i * ep.ldy] = at(i, piece)[c];
              }
            }
          }
        }
        __syncwarp();
        if (shifted) {
          // Plain rows off the 16-byte grid (an odd vocabulary): the 16-byte pieces of the row's memory lie s values into those of the
          // block.  A lane takes its piece and its neighbour's and shifts out the eight values that one store takes; the s values
          // ahead of the first such piece and the 8 - s behind the last are stored singly (834 x 50257 x 512 60 -> 52 us).
          const int piece = lane & 7, r0 = lane >> 3;
          const size_t base = (reinterpret_cast<uintptr_t>(ep.y) >> 1) + nb;
#pragma unroll
          for (int i = 0; i < 8; i++) {
            const int row = r0 + i * 4;
            const size_t off = (size_t)(first + row) * ep.ldy;
            const int s = (int)(8 - ((base + off) & 7)) & 7;
            const uint4 v = *reinterpret_cast<const uint4*>(at(row, piece));
            uint32_t w[8] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int j = 0; j < 4; j++) w[4 + j] = __shfl_down_sync(0xffffffffu, w[j], 1);
#pragma unroll
            for (int j = 0; j < 6; j++) w[j] = s & 4 ? w[j + 2] : w[j];
#pragma unroll
            for (int j = 0; j < 5; j++) w[j] = s & 2 ? w[j + 1] : w[j];
#pragma unroll
            for (int j = 0; j < 4; j++) w[j] = __funnelshift_r(w[j], w[j + 1], s & 1 ? 16 : 0);
            if (row < rows && (s == 0 || piece < 7))
              *reinterpret_cast<uint4*>(ep.y + off + nb + piece * 8 + s) = make_uint4(w[0], w[1], w[2], w[3]);
          }
#pragma unroll
          for (int i = 0; i < 8; i++) {
            const int row = i * 4 + (lane >> 3), j = lane & 7;
            const size_t off = (size_t)(first + row) * ep.ldy;
            const int s = (int)(8 - ((base + off) & 7)) & 7;
            const int col = j < s ? j : 56 + j;
            if (row < rows && s != 0) ep.y[off + nb + col] = at(row, col >> 3)[col & 7];
          }
        }
        if (!unaligned) {
          const int piece = lane & 7, r0 = lane >> 3;   // 8 values of row r0, r0 + 4, ...
          const int n = nb + piece * 8;
          if (EPI == EPI_HIST_T) {
            const int nt = nb + (piece & 3) * 16;   // first of the 16 tokens whose even or odd half this is
            if (nt < N) {
              const int b = nt / ep.Tseq, t = ep.t0 + (nt - b * ep.Tseq);
              bf16* yc = ep.y + (((size_t)b * ep.ldy + first) * 2 + (piece >> 2)) * ep.Lh + (t >> 1);
#pragma unroll
              for (int i = 0; i < 8; i++)
                if (r0 + i * 4 < rows)
                  *reinterpret_cast<uint4*>(yc + (size_t)(r0 + i * 4) * 2 * ep.Lh) =
                      *reinterpret_cast<const uint4*>(at(r0 + i * 4, piece));
            }
          } else if (n + 8 <= N) {
            bf16* yc = ep.y + (size_t)(first + r0) * ep.ldy +
                       (EPI == EPI_BLOCKCOL ? (size_t)(n / ep.Tseq) * ep.ld2 + n % ep.Tseq : (size_t)n);   // Tseq % 8 == 0
            if (EPI == EPI_RESID) {
              const bf16* rc = ep.resid + (size_t)(first + r0) * ep.ldr + n;
              uint4 res[8];
#pragma unroll
              for (int i = 0; i < 8; i++)
                res[i] = r0 + i * 4 < rows ? *reinterpret_cast<const uint4*>(rc + (size_t)(i * 4) * ep.ldr)
                                           : make_uint4(0, 0, 0, 0);
#pragma unroll
              for (int i = 0; i < 8; i++)
                if (r0 + i * 4 < rows) {
                  float o[8], rs[8];
                  load_vec(at(r0 + i * 4, piece), o);
                  load_vec(reinterpret_cast<const bf16*>(&res[i]), rs);
#pragma unroll
                  for (int j = 0; j < 8; j++) o[j] += rs[j];
                  store_vec(yc + (size_t)(i * 4) * ep.ldy, o);
                }
            } else {
#pragma unroll
              for (int i = 0; i < 8; i++)
                if (r0 + i * 4 < rows)
                  *reinterpret_cast<uint4*>(yc + (size_t)(i * 4) * ep.ldy) =
                      *reinterpret_cast<const uint4*>(at(r0 + i * 4, piece));
            }
          } else {   // the last columns of a width that is no multiple of 8
            for (int j = n; j < min(n + 8, N); j++)
              for (int i = r0; i < rows; i += 4) {
                const bf16 v = at(i, piece)[j - n];
                const size_t m = (size_t)(first + i);
                if (EPI == EPI_RESID)
                  ep.y[m * ep.ldy + j] = __float2bfloat16_rn(__bfloat162float(ep.resid[m * ep.ldr + j]) + __bfloat162float(v));
                else if (EPI == EPI_BLOCKCOL)
                  ep.y[m * ep.ldy + (size_t)(j / ep.Tseq) * ep.ld2 + j % ep.Tseq] = v;
                else
                  ep.y[m * ep.ldy + j] = v;
              }
          }
        }
        __syncwarp();   // the block has been read
      }
      // this warp's TMEM reads of the buffer are complete (wait::ld above): hand it back to the pair's MMA warp
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(hand_back + buf * (uint32_t)sizeof(uint64_t));
    }
    if (COPIES && lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");   // (none where nothing was sent)
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  }
  __syncwarp();
  __syncthreads();
  if constexpr (PAIR) {
    if (threadIdx.x == 0 && *abort_flag) {   // tell the other CTA
      store_to_cta(abort_flag + 1, rank ^ 1, 1);
      asm volatile("fence.acq_rel.cluster;" ::: "memory");
    }
    __syncwarp();
    pair_sync();   // neither CTA leaves while the other's instructions, copies' barriers or arrivals still use its memory
  }
  if (abort_flag[0] || abort_flag[1]) {
    // A wait ran out.  Report it, then let copies that were issued but never consumed land (bounded)
    // before either CTA's shared memory is released.
    if (rank == 0 && threadIdx.x == 0) {
      if (status) atomicExch(status, 3);
      const int issued = PAIR ? max(*issued_ctr, (int)load_from_cta(issued_ctr, 1)) : *issued_ctr, consumed = *consumed_ctr;
      const uint64_t drain_start = global_ns();
      for (int g = consumed; g < issued; g++) {
        const int s = g % STAGES;
        const uint32_t ph = (uint32_t)(g / STAGES) & 1u;
        for (uint32_t w = 0; w < WAIT_LIMIT; ++w) {
          if (mbar_try_wait(&full_bar[s], ph)) break;
          if ((w & 255u) == 255u && global_ns() - drain_start > wait_ns) break;
        }
      }
    }
    __syncwarp();
    if constexpr (PAIR) pair_sync();
    else __syncthreads();
  }
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if constexpr (PAIR) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS));
    else asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS));
  }
}

// The split tiles' sums over their parts, first to last, and the epilogue.  A CTA: 8 rows x 128 columns of a tile, a thread 4 columns (8 rows x 16 bytes of a
// part are 128 bytes in a row, 4 threads' outputs 32 bytes of theirs).
template <int EPI>
__global__ void __launch_bounds__(256) split_sum_kernel(const float* __restrict__ partials, int whole, int parts, int M, int N, int tiles_m, int tiles_n,
                                                        int group_m, EpiArgs<bf16> ep) {
  pdl_wait();
  pdl_trigger();
  int tm, tn;
  tile_coords(whole + blockIdx.y, tiles_m, tiles_n, group_m, tm, tn);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int row = (blockIdx.x >> 1) * 8 + (lane & 7), c4 = (blockIdx.x & 1) * 32 + warp * 4 + (lane >> 3);
  const int m = tm * 256 + row, n = tn * 256 + c4 * 4;
  if (m >= M || n >= N) return;
  const float4* p = reinterpret_cast<const float4*>(partials + (size_t)blockIdx.y * SPLIT_TILE) + ((row >> 5) * 64 + c4) * 32 + (row & 31);
  float4 acc = __ldcs(p);
#pragma unroll 8
  for (int i = 1; i < parts; i++) {
    const float4 v = __ldcs(p + (size_t)i * gridDim.y * (SPLIT_TILE / 4));
    acc.x += v.x, acc.y += v.y, acc.z += v.z, acc.w += v.w;
  }
  const float o[4] = {acc.x, acc.y, acc.z, acc.w};
  const bool vec = n + 4 <= N && ep.ldy % 4 == 0 && (reinterpret_cast<uintptr_t>(ep.y) & 7) == 0;
  bf16* y = ep.y + (size_t)m * ep.ldy + n;
  if (EPI == EPI_RESID) {   // rows of resid and y on the 16-byte grid (gemm_tc_supported)
    const bf16* rr = ep.resid + (size_t)m * ep.ldr + n;
    for (int j = 0; j < min(4, N - n); j++)
      if (!vec) y[j] = __float2bfloat16_rn(__bfloat162float(rr[j]) + round_to<bf16>(o[j]));
    if (vec) {
      const uint2 rv = *reinterpret_cast<const uint2*>(rr);
      const float r[4] = {__uint_as_float(rv.x << 16), __uint_as_float(rv.x & 0xffff0000u), __uint_as_float(rv.y << 16),
                          __uint_as_float(rv.y & 0xffff0000u)};
      const __nv_bfloat162 a = __floats2bfloat162_rn(r[0] + round_to<bf16>(o[0]), r[1] + round_to<bf16>(o[1]));
      const __nv_bfloat162 b = __floats2bfloat162_rn(r[2] + round_to<bf16>(o[2]), r[3] + round_to<bf16>(o[3]));
      *reinterpret_cast<uint2*>(y) = make_uint2(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&b));
    }
  } else if (vec) {
    const __nv_bfloat162 a = __floats2bfloat162_rn(o[0], o[1]), b = __floats2bfloat162_rn(o[2], o[3]);
    *reinterpret_cast<uint2*>(y) = make_uint2(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&b));
  } else {
    for (int j = 0; j < min(4, N - n); j++) y[j] = __float2bfloat16_rn(o[j]);
  }
}

// ---------------------------------------------------------------------------------------------- host
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn get_encode_fn() {
  static EncodeTiledFn fn = nullptr;
  static bool tried = false;
  if (!tried) {
    tried = true;
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = (EncodeTiledFn)p;
  }
  return fn;
}

// 2-D map over a row-major bf16 matrix [rows, cols] with row stride ld (elements); box 64 x box_rows, 128B swizzle.
// A map depends on nothing but these arguments, so the encoded maps are kept in a small per-thread table keyed by
// them (a token step asks for the same few dozen maps over and over; an entry never goes stale, it is just an address
// and a shape).
struct MapKey {
  const void* base;
  long long rows, cols, ld;
  int box_rows;
  bool operator==(const MapKey& o) const {
    return base == o.base && rows == o.rows && cols == o.cols && ld == o.ld && box_rows == o.box_rows;
  }
};
struct MapSlot {
  MapKey key;
  CUtensorMap map;
  bool used;
};
constexpr int MAP_SLOTS = 1024;   // direct-mapped
int make_map_uncached(CUtensorMap* map, const void* base, long long rows, long long cols, long long ld, int box_rows);
int make_map(CUtensorMap* map, const void* base, long long rows, long long cols, long long ld, int box_rows = BM) {
  static thread_local MapSlot* table = nullptr;
  if (!table) table = new MapSlot[MAP_SLOTS]();
  const MapKey key{base, rows, cols, ld, box_rows};
  unsigned long long h = (unsigned long long)(uintptr_t)base * 0x9E3779B97F4A7C15ull;
  h ^= (unsigned long long)rows * 0xC2B2AE3D27D4EB4Full + (unsigned long long)cols * 0x165667B19E3779F9ull +
       (unsigned long long)ld * 0x27D4EB2F165667C5ull + (unsigned long long)box_rows;
  MapSlot& slot = table[(h >> 20) % MAP_SLOTS];
  if (slot.used && slot.key == key) {
    *map = slot.map;
    return STU_OK;
  }
  const int rc = make_map_uncached(map, base, rows, cols, ld, box_rows);
  if (rc == STU_OK) {
    slot.key = key;
    slot.map = *map;
    slot.used = true;
  }
  return rc;
}
int make_map_uncached(CUtensorMap* map, const void* base, long long rows, long long cols, long long ld, int box_rows) {
  EncodeTiledFn fn = get_encode_fn();
  if (!fn) return STU_ERR_UNSUPPORTED;
  cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)ld * 2};
  cuuint32_t box[2] = {(cuuint32_t)BK, (cuuint32_t)box_rows};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? STU_OK : STU_ERR_UNSUPPORTED;
}

// The same over an output, boxes of 32 rows x 64 columns: rows of ldy elements, or (column blocks) blocks of Tseq columns ld2 apart.
int make_output_map(CUtensorMap* map, const EpiArgs<bf16>& ep, bool blocks, int M, int N) {
  EncodeTiledFn fn = get_encode_fn();
  if (!fn) return STU_ERR_UNSUPPORTED;
  const cuuint64_t dims[3] = {(cuuint64_t)(blocks ? ep.Tseq : N), (cuuint64_t)M, (cuuint64_t)(blocks ? N / ep.Tseq : 1)};
  const cuuint64_t strides[2] = {(cuuint64_t)ep.ldy * 2, (cuuint64_t)ep.ld2 * 2};
  const cuuint32_t box[3] = {64, 32, 1}, estr[3] = {1, 1, 1};
  const CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, blocks ? 3 : 2, ep.y, dims, strides, box, estr,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_NONE,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? STU_OK : STU_ERR_UNSUPPORTED;
}

// Failure-detection test hooks (stu_test_inject_wait_expiry): drop the first operand copy of the next launch, and the
// wall-time bound of every mbarrier wait.
int g_drop_first_copy = 0;
unsigned long long g_wait_ns = 2000000000ull;

// Row by row while the whole B operand stays in L2 (up to 48 MB, a share of the 126 MB that the rows of A and the
// output leave alone) or has so few column tiles that the tiles in flight cover several row tiles anyway.  Otherwise
// bands of 16 row tiles of 256: a wave then reads 16 * 256 rows of A and few column tiles instead of all of B.  us, row by row and bands
// of 8, 16, 32: gate/up 32768 x 12288 x 3072 4547, 3608, 3620, 3796; 32768 x 9216 x 3072 1413, 1406, 1354, 1415; 7996 x 50257 x 1024 967, 750,
// 736, 725.  Below the lines bands of 16 cost 0 (gate/up of d = 1536) to 7 % (65536 x 1536 x 6144).
int gemm_group_m(int tiles_n, int N, int K, bool dual) {
  return tiles_n > 24 && (long long)N * K * (dual ? 4 : 2) > (48ll << 20) ? 16 : 1;
}

template <int EPI, int STAGES, int TN, int CTAS>
constexpr size_t tc_smem() {
  constexpr bool DUAL = (EPI == EPI_GELU_MUL);
  constexpr size_t stage = (size_t)stage_blocks(DUAL ? 2 * TN : TN) * (A_BYTES + (DUAL ? 2 * TN : TN) / CTAS * BK * 2);
  constexpr size_t bytes = STAGES * stage + 1024 + 1024 + EPI_WARPS * BLOCK_BYTES;
  static_assert(bytes > 114 * 1024 && bytes <= 227 * 1024, "one CTA per SM, whatever the form: device_pairs");
  return bytes;
}

// Pairs of CTAs that the current device runs at a time (every form of the kernel fills an SM).
int device_pairs() {
  static std::atomic<int> found[STU_MAX_DEVICES] = {};
  std::atomic<int>& n = found[current_device()];
  if (n.load(std::memory_order_relaxed) == 0) {
    const void* kernel = (const void*)gemm_tc_kernel<EPI_STORE, 6, 256, 2, false>;
    constexpr size_t smem = tc_smem<EPI_STORE, 6, 256, 2>();
    static SmemLimit limit;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2 * device_sm_count());
    cfg.blockDim = dim3(64 + 32 * EPI_WARPS);
    cfg.dynamicSmemBytes = smem;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = 2;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    int clusters = 0;
    if (allow_smem(kernel, smem, limit) != cudaSuccess || cudaOccupancyMaxActiveClusters(&clusters, kernel, &cfg) != cudaSuccess || clusters < 1) {
      (void)cudaGetLastError();
      clusters = device_sm_count() / 2;
    }
    n.store(clusters, std::memory_order_relaxed);
  }
  return n.load(std::memory_order_relaxed);
}

template <int EPI, int STAGES, int TN, int CTAS = 2, bool SPLIT = false>
int launch_tc(const CUtensorMap& a, const CUtensorMap& b, const CUtensorMap& b2, int M, int N, int K, int m_fast,
              int causal, const EpiArgs<bf16>& ep, int* status, cudaStream_t st, SplitK split = {}) {
  constexpr bool DUAL = (EPI == EPI_GELU_MUL);
  constexpr bool COPIES = (EPI == EPI_STORE || EPI == EPI_GELU_MUL || EPI == EPI_BLOCKCOL);
  constexpr size_t smem = tc_smem<EPI, STAGES, TN, CTAS>();
  // The output by tensor copies: rows on the 16-byte grid and of whole 16 bytes (a copy clips at those), and (column blocks) 64
  // columns inside one block of a whole number of them.  What gains is many outputs for little K: LDS features, 6144 x 48128 x
  // 320, 237 -> 204 us; products of K = 1024 and more hide either form.
  CUtensorMap y = a;
  int by_copy = 0;
  if (COPIES && !ep.peer && ep.ldy % 8 == 0 && N % 8 == 0 && aligned16(ep.y) && (EPI != EPI_BLOCKCOL || (ep.Tseq % 64 == 0 && N % ep.Tseq == 0)))
    by_copy = make_output_map(&y, ep, EPI == EPI_BLOCKCOL, M, N) == STU_OK;
  auto k = gemm_tc_kernel<EPI, STAGES, TN, CTAS, SPLIT>;
  static SmemLimit limit;
  cudaError_t e = allow_smem((const void*)k, smem, limit);
  if (e != cudaSuccess) return (int)e;
  const int tiles_m = (M + CTAS * BM - 1) / (CTAS * BM), tiles_n = (N + TN - 1) / TN;
  const int tiles = SPLIT ? split.whole + (tiles_m * tiles_n - split.whole) * split.parts : tiles_m * tiles_n, most = CTAS == 2 ? device_pairs() : device_sm_count();
  const int grid = CTAS * (tiles < most ? tiles : most);  // one persistent CTA per SM
  const int drop = take_dropped_stage();
  const int group_m = m_fast ? tiles_m : gemm_group_m(tiles_n, N, K, DUAL);
  e = launch_maybe_overlapped(k, dim3(grid), dim3(64 + 32 * EPI_WARPS), smem, st, true, a, b, b2, y, by_copy, M, N, K, tiles_m, tiles_n, group_m,
                              causal, ep, status, drop, g_wait_ns, split);
  if (e != cudaSuccess) return (int)e;
  STU_CHECK_LAUNCH();
  if constexpr (SPLIT) {
    e = launch_maybe_overlapped(split_sum_kernel<EPI>, dim3(64, tiles_m * tiles_n - split.whole), dim3(256), 0, st, true, (const float*)split.partials,
                                split.whole, split.parts, M, N, tiles_m, tiles_n, group_m, ep);
    if (e != cudaSuccess) return (int)e;
    STU_CHECK_LAUNCH();
    t_linear_launches = 2;
  }
  return STU_OK;
}

// ------------------------------------------------------------------------------------------------
// Token-step linear layers for 9..64 activation rows on the tensor cores, operands swapped: the WEIGHTS are the
// 128-row operand (a tile = 128 output features, or 64 gate + 64 up rows of the same 64 features), the activation rows
// the 16-, 32- or 64-column one, so every weight byte passes through shared memory exactly once and goes straight into
// tcgen05.mma (M = 128, N = 32, K = 16); nothing is staged through registers and there is no cross-warp reduction.
// The K range is split over the CTAs of a thread-block cluster (up to 16; grid = tiles x KSPLIT, about one to two CTAs per SM,
// 80 KB of operands in flight each); every CTA drains its 128 x 32 fp32 accumulator from tensor memory into its own
// shared memory (token-major, conflict-free), the cluster synchronises, and every CTA sums the partial tiles of its
// share of the tokens in a fixed order through distributed shared memory and runs their epilogue (coalesced along
// the features).
// Launched with the programmatic attribute: the successor is released once tensor memory has been allocated (a
// co-resident successor that allocated first could otherwise block this kernel's allocation while waiting for it), in gate/up and
// without early_weights once the kernel in front is complete (PdlTrigger, epilogue.cuh);
// with early_weights (the caller's promise that the preceding kernel does not write the weights) the weight tiles of
// the first stages are requested before griddepcontrol.wait, the activation tiles after it.

// SU_BN: activation rows per tile, 16, 32 or 64 (the N of the MMA, the accumulator's columns).  nstages: ring depth,
// chosen by the host: shallow (two CTAs per SM) for grids of more CTAs than SMs, deep below that.
// (A fused RMSNorm - the drain warps normalising the rows into swizzled shared-memory tiles while the weight stream
// runs, bit-identical to the norm kernel - was built and measured: the 24-layer token step went from 1.71-1.85 ms
// to 2.12-2.25 ms, the MMAs waiting for 32 rows of statistics that a separate, overlapped norm kernel has long
// finished.  Callers keep the separate norm kernel.)
constexpr int SU_MAXST = 10;
template <int EPI, int KSPLIT, int SU_BN>
__global__ void __launch_bounds__(192, 1)
    skinny_umma_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmW2,
                       const __grid_constant__ CUtensorMap tmX, int M, int N, int K, EpiArgs<bf16> ep, int* status,
                       int early_weights, unsigned long long wait_ns, int nstages) {
  constexpr bool DUAL = (EPI == EPI_GELU_MUL);
  constexpr int NF = DUAL ? 64 : 128;   // output features per tile
  constexpr int SU_B_BYTES = SU_BN * BK * 2;
  constexpr int PART_BYTES = SU_BN * BM * 4;
  constexpr int stage_bytes = A_BYTES + SU_B_BYTES;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n0 = blockIdx.x * NF;
  const int num_kb = (K + BK - 1) / BK;
  const int per = (num_kb + KSPLIT - 1) / KSPLIT;
  const int kb0 = (int)blockIdx.y * per;
  const int nkb = max(0, min(num_kb, kb0 + per) - kb0);
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  // ring | partial tile | barriers
  float* part = reinterpret_cast<float*>(smem + nstages * stage_bytes);   // [SU_BN tokens][128 rows]
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + nstages * stage_bytes + PART_BYTES);
  uint64_t* empty_bar = full_bar + SU_MAXST;
  uint64_t* tmem_full = empty_bar + SU_MAXST;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tmem_full + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  int* issued_ctr = const_cast<int*>(reinterpret_cast<volatile int*>(tmem_slot + 2));
  int* consumed_ctr = issued_ctr + 1;

  if (threadIdx.x == 0) {
    for (int s = 0; s < nstages; s++) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    mbar_init(tmem_full, 1);
    *abort_flag = 0;
    *issued_ctr = 0;
    *consumed_ctr = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"(SU_BN < 32 ? 32 : SU_BN));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::);
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_base = *tmem_slot;
  const bool early_trigger = early_weights && PdlTrigger<EPI>::ahead_of_wait;
  if (early_trigger) pdl_trigger();   // only now: this CTA holds its tensor memory

  if (warp == 0) {
    // ---------------- TMA producer
    const bool leader = elect_one();
    auto load_w = [&](int s, int kb) {
      unsigned char* sa = smem + s * stage_bytes;
      if (DUAL) {   // 64 gate rows, then the 64 up rows of the same features
        tma_load_2d(sa, &tmW, &full_bar[s], kb * BK, n0);
        tma_load_2d(sa + A_BYTES / 2, &tmW2, &full_bar[s], kb * BK, n0);
      } else {
        tma_load_2d(sa, &tmW, &full_bar[s], kb * BK, n0);
      }
    };
    auto load_x = [&](int s, int kb) {
      tma_load_2d(smem + s * stage_bytes + A_BYTES, &tmX, &full_bar[s], kb * BK, 0);
    };
    const int pre = early_weights ? min(nstages, nkb) : 0;
    for (int g = 0; g < pre; g++)
      if (leader) {
        mbar_expect_tx(&full_bar[g], stage_bytes);
        load_w(g, kb0 + g);
      }
    pdl_wait();   // the activations are the output of the kernel before this one
    if (!early_trigger) pdl_trigger();
    for (int g = 0; g < pre; g++)
      if (leader) load_x(g, kb0 + g);
    int g = pre, s = pre == nstages ? 0 : pre;
    uint32_t ph = pre == nstages ? 0u : 1u;
    for (; g < nkb; g++) {
      if (!warp_wait(&empty_bar[s], ph, abort_flag, wait_ns)) break;
      if (leader) {
        mbar_expect_tx(&full_bar[s], stage_bytes);
        load_w(s, kb0 + g);
        load_x(s, kb0 + g);
      }
      if (++s == nstages) s = 0, ph ^= 1u;
    }
    if (leader) *issued_ctr = g;
  } else if (warp == 1) {
    // ---------------- MMA issuer
    const bool leader = elect_one();
    const uint64_t da0 = make_smem_desc(smem_u32(smem)), db0 = make_smem_desc(smem_u32(smem) + A_BYTES);
    bool ok = true;
    int g = 0, s = 0;
    uint32_t ph = 0;
    for (; g < nkb; g++) {
      ok = warp_wait(&full_bar[s], ph, abort_flag, wait_ns);
      if (!ok) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      if (leader) {
        const uint64_t da = da0 + (uint64_t)(s * (stage_bytes >> 4)), db = db0 + (uint64_t)(s * (stage_bytes >> 4));
#pragma unroll
        for (int kk = 0; kk < BK / 16; kk++) umma<SU_BN>(tmem_base, da + 2 * kk, db + 2 * kk, (g | kk) ? 1u : 0u);
        if (g + nstages < nkb) umma_commit(&empty_bar[s]);   // (nobody waits for the last round's)
        if (g + 1 == nkb) umma_commit(tmem_full);
      }
      __syncwarp();
      if (++s == nstages) s = 0, ph ^= 1u;
    }
    if (leader) *consumed_ctr = g;
  } else {
    // ---------------- accumulator drain: TMEM lane quarter = warp % 4, one weight row per thread
    const int quarter = warp & 3;
    const int row = quarter * 32 + lane;
    bool ok = true;
    if (nkb > 0) {
      ok = mbar_wait(tmem_full, 0, abort_flag, wait_ns);
      ok = __all_sync(0xffffffffu, ok);
      if (ok) asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    }
#pragma unroll
    for (int h = 0; h < (SU_BN + 31) / 32; h++) {   // 16 rows: 32 columns are allocated, the upper 16 unused
      uint32_t r[32];
#pragma unroll
      for (int c = 0; c < 32; c++) r[c] = 0u;
      if (nkb > 0 && ok) {
        tmem_ld32(tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(h * 32), r);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
      }
#pragma unroll
      for (int c = 0; c < (SU_BN < 32 ? SU_BN : 32); c++) part[(h * 32 + c) * BM + row] = __uint_as_float(r[c]);
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  }
  // ---- the partial tiles of the cluster meet (the role branches left the warps of the producer and of the MMA
  // issuer diverged: they reconverge before the aligned cluster barrier)
  __syncwarp();
  __syncthreads();
  cg::cluster_group cluster = cg::this_cluster();
  if constexpr (KSPLIT > 1) cluster.sync();
  {
    // every CTA of the cluster sums and stores the tokens rank, rank + KSPLIT, ... of the tile (fixed order of the
    // partial tiles, whoever sums them)
    pdl_wait();   // returns at once (the producer waited before the first activation copy)
    const int rank = KSPLIT > 1 ? (int)cluster.block_rank() : 0;
    const float* parts[KSPLIT];
#pragma unroll
    for (int rk = 0; rk < KSPLIT; rk++) parts[rk] = KSPLIT > 1 ? cluster.map_shared_rank(part, rk) : part;
    auto sum_at = [&](int idx) {
      float v = parts[0][idx];
#pragma unroll
      for (int rk = 1; rk < KSPLIT; rk++) v += parts[rk][idx];
      return v;
    };
    if (!*abort_flag) {
      for (int e = threadIdx.x; e < ((SU_BN + KSPLIT - 1) / KSPLIT) * NF; e += 192) {
        const int mi = e / NF, f = e - mi * NF, m = rank + mi * KSPLIT, n = n0 + f;
        if (m < M && m < SU_BN && n < N)
          epilogue_store<bf16, EPI>(ep, m, n, sum_at(m * BM + f), DUAL ? sum_at(m * BM + 64 + f) : 0.f);
      }
    }
  }
  if constexpr (KSPLIT > 1) cluster.sync(); else __syncthreads();   // the other CTAs' partial tiles stay alive until read
  if (*abort_flag) {
    if (threadIdx.x == 0) {
      if (status) atomicExch(status, 3);
      const int issued = *issued_ctr, consumed = *consumed_ctr;
      const uint64_t drain_start = global_ns();
      for (int g = consumed; g < issued; g++) {
        const int s = g % nstages;
        const uint32_t ph = (uint32_t)(g / nstages) & 1u;
        for (uint32_t w = 0; w < WAIT_LIMIT; ++w) {
          if (mbar_try_wait(&full_bar[s], ph)) break;
          if ((w & 255u) == 255u && global_ns() - drain_start > wait_ns) break;
        }
      }
    }
    __syncthreads();
  }
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(SU_BN < 32 ? 32 : SU_BN));
  }
}

// Shared memory of one CTA: ring, partial tile, barriers and bookkeeping, alignment slack.
template <int SU_BN>
size_t su_smem_bytes(int nstages) {
  return (size_t)nstages * (A_BYTES + SU_BN * BK * 2) + (size_t)SU_BN * BM * 4 + (2 * SU_MAXST + 1) * 8 + 64 + 1024;
}

template <int EPI, int KSPLIT, int SU_BN>
int launch_skinny_umma(const CUtensorMap& w, const CUtensorMap& w2, const CUtensorMap& x, int M, int N, int K,
                       const EpiArgs<bf16>& ep, int early, int* status, cudaStream_t st) {
  constexpr int NF = (EPI == EPI_GELU_MUL) ? 64 : 128;
  const int tiles = (N + NF - 1) / NF;
  // ring depth: deep (about 160 KB of weights in flight, one CTA per SM) for grids that leave a third of the SMs
  // empty anyway, else as deep as lets two CTAs share an SM
  bool deep = 3 * tiles * KSPLIT <= 2 * device_sm_count();
  if (const char* sv = getenv("STU_B200_UMMA_STAGES")) deep = atoi(sv) == 8;   // tuning aid
  const size_t two_per_sm = (233472 / 2) - 1024;   // per-SM shared memory, per-CTA reservation
  int nstages = deep ? (SU_BN == 16 ? 10 : (SU_BN == 32 ? 8 : 6)) : 2;
  if (!deep)
    while (nstages < SU_MAXST && su_smem_bytes<SU_BN>(nstages + 1) <= two_per_sm) nstages++;
  while (nstages > 2 && su_smem_bytes<SU_BN>(nstages) > 227 * 1024) nstages--;
  if (su_smem_bytes<SU_BN>(nstages) > 227 * 1024) return STU_ERR_UNSUPPORTED;
  if (!deep && nstages > 5) nstages = 5;
  const size_t smem = su_smem_bytes<SU_BN>(nstages);
  auto kern = skinny_umma_kernel<EPI, KSPLIT, SU_BN>;
  static SmemLimit limit;
  cudaError_t e = allow_smem((const void*)kern, smem, limit);
  if (e != cudaSuccess) return (int)e;
  if (KSPLIT > 8) {   // clusters of 16 CTAs are outside the portable range
    e = cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e != cudaSuccess) return (int)e;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(tiles, KSPLIT);
  cfg.blockDim = dim3(192);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = 1;
  at[0].val.clusterDim.y = KSPLIT;
  at[0].val.clusterDim.z = 1;
  at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  static std::atomic<int> cosched[STU_MAX_DEVICES] = {};   // the most shared memory per CTA that was found to fit
  const int dev = current_device();
  if (KSPLIT > 8 && cosched[dev].load(std::memory_order_relaxed) < (int)smem) {   // can the GPU co-schedule a cluster of this size and footprint at all?  (the caller falls back)
    int clusters = 0;
    if (cudaOccupancyMaxActiveClusters(&clusters, kern, &cfg) != cudaSuccess || clusters < 1) {
      (void)cudaGetLastError();
      return STU_ERR_UNSUPPORTED;
    }
    cosched[dev].store((int)smem, std::memory_order_relaxed);
  }
  cfg.numAttrs = pdl_enabled() ? 2 : 1;
  e = cudaLaunchKernelEx(&cfg, kern, w, w2, x, M, N, K, ep, status, early, g_wait_ns, nstages);
  if (e != cudaSuccess) return (int)e;
  STU_CHECK_LAUNCH();
  return STU_OK;
}

template <int EPI, int KSPLIT>
int launch_skinny_umma_bn(const CUtensorMap& w, const CUtensorMap& w2, const CUtensorMap& x, int M, int N, int K,
                          const EpiArgs<bf16>& ep, int early, int* status, cudaStream_t st) {
  if (M <= 16) return launch_skinny_umma<EPI, KSPLIT, 16>(w, w2, x, M, N, K, ep, early, status, st);
  if (M <= 32) return launch_skinny_umma<EPI, KSPLIT, 32>(w, w2, x, M, N, K, ep, early, status, st);
  return launch_skinny_umma<EPI, KSPLIT, 64>(w, w2, x, M, N, K, ep, early, status, st);
}

template <int EPI>
int launch_skinny_umma_split(int ks, const CUtensorMap& w, const CUtensorMap& w2, const CUtensorMap& x, int M, int N,
                             int K, const EpiArgs<bf16>& ep, int early, int* status,
                             cudaStream_t st) {
  switch (ks) {
    case 1: return launch_skinny_umma_bn<EPI, 1>(w, w2, x, M, N, K, ep, early, status, st);
    case 2: return launch_skinny_umma_bn<EPI, 2>(w, w2, x, M, N, K, ep, early, status, st);
    case 4: return launch_skinny_umma_bn<EPI, 4>(w, w2, x, M, N, K, ep, early, status, st);
    case 16: {
      const int rc = launch_skinny_umma_bn<EPI, 16>(w, w2, x, M, N, K, ep, early, status, st);
      if (rc != STU_ERR_UNSUPPORTED) return rc;   // no room for clusters of 16 on this GPU: clusters of 8
    }
      [[fallthrough]];
    default: return launch_skinny_umma_bn<EPI, 8>(w, w2, x, M, N, K, ep, early, status, st);
  }
}

}  // namespace

// Per-device state of the library: the status word the host wrapper registered for the device that was current at
// the time (a kernel must never be handed a word that lives on another GPU) and that device's SM count.
static int* g_status_words[STU_MAX_DEVICES] = {nullptr};
static int g_sm_counts[STU_MAX_DEVICES] = {0};

static int current_device() {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= STU_MAX_DEVICES) return 0;
  return dev;
}

int device_sm_count() {
  const int dev = current_device();
  int n = g_sm_counts[dev];
  if (n <= 0) {
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 148;
    g_sm_counts[dev] = n;
  }
  return n;
}

int* device_status_word() { return g_status_words[current_device()]; }

// Test hook for the failure-detection path: the next launch of this process of a tcgen05 GEMM (bf16 or fp32), of the full variant's fp32 convolutions or of
// its token step on tcgen05 never fills its first pipeline stage, and every bounded wait of theirs gives up after wait_ms milliseconds (0 restores
// the default of two seconds without arming a fault).  The kernel then reports its status, drains what it did issue, frees its tensor
// memory and returns; nothing faults and the context stays usable.
extern "C" int stu_test_inject_wait_expiry(int wait_ms) {
  if (wait_ms < 0 || wait_ms > 10000) return STU_ERR_SHAPE;
  if (wait_ms == 0) {
    g_drop_first_copy = 0;
    g_wait_ns = 2000000000ull;
  } else {
    g_drop_first_copy = 1;
    g_wait_ns = (unsigned long long)wait_ms * 1000000ull;
  }
  return STU_OK;
}

unsigned long long wait_bound_ns() { return g_wait_ns; }
bool take_dropped_stage() {   // the injected fault applies to one launch
  const bool drop = g_drop_first_copy != 0;
  g_drop_first_copy = 0;
  return drop;
}

// make_map for the other tensor-core kernels of K-major bf16 operands.
int operand_map(CUtensorMap* map, const void* base, long long rows, long long cols, long long ld, int box_rows) {
  return make_map(map, base, rows, cols, ld, box_rows);
}

extern "C" int stu_set_status_word(int* device_status) {
  g_status_words[current_device()] = device_status;
  return STU_OK;
}

bool gemm_tc_supported(const void* A, long long lda, const void* B, long long ldb, long long skb, const void* B2,
                       int M, int N, int K, int epi, const EpiArgsAny& ep, int dtype) {
  if (dtype != STU_BF16 || skb != 1) return false;
  static const bool disabled = getenv("STU_B200_DISABLE_TCGEN05") != nullptr;  // debugging aid: CUDA-core GEMM instead
  if (disabled) return false;
  if (lda % 8 || ldb % 8 || K % 8 || !aligned16(A) || !aligned16(B) || (B2 && !aligned16(B2))) return false;
  if (M < 1 || N < 1 || K < 8) return false;
  if (epi == EPI_HIST) return aligned16(ep.y) && get_encode_fn() != nullptr;
  if (epi != EPI_STORE && (ep.ldy % 8 || !aligned16(ep.y))) return false;   // plain stores take any row stride
  if (epi == EPI_BLOCKCOL && (ep.ld2 % 8 || ep.Tseq % 8 || ep.Tseq <= 0)) return false;
  if (epi == EPI_RESID && (ep.ldr % 8 || !aligned16(ep.resid))) return false;
  return get_encode_fn() != nullptr;
}

// 256-column tiles where their waves over the pairs of SMs take less time than those of 128 columns: a wide tile costs 1.74
// narrow ones where all pairs are busy (65536 x 1536 x 6144, 21 waves against 42: 900 and 1034 us; 1.87 where only one pair is:
// 256 rows, K = 16384, 76.5 and 41.0).  One wave of either, 1668 x 768 x 3072: narrow 12.0 us, wide 18.3; two wide ones against
// four narrow, 7996 x 1024 x 4096: 66.6 and 58.7.
// Tiles of 128 x 256 by single CTAs where those of 256 rows fill their last wave badly (M mod 256 up to 128, one wave against two): a wave of
// them costs 1.10 to 1.17 of the pairs' wide ones (shared memory, see the head of this file), counted as 1.24 because it gains less
// than its waves say where there are many.  us, pairs and single: gate/up 300 x 6144 x 1536 20.5 and 15.0 (1 wave for 2), 100 x 10240 x 2560 32.6 and
// 24.6, 300 x 12288 x 3072 55.6 and 51.6 (2 for 3), 1030 x 6144 x 1536 43.4 and 40.4 (3 for 4), 1030 x 12288 x 3072 127 and 137 (6 for 7: pairs);
// plain 300 x 12288 x 4096 45.9 and 34.8, 1030 x 7680 x 2560 42.7 and 36.9, 300 x 50257 x 2560 102 and 92; residual 3661 x 2560 x 10240 196 and 152;
// with as many waves 7996 x 4096 x 1024 gate/up 108 and 129.  (16.7, 26.6, 50.9, 41.0, 130; 34.3, 37.4, 94; 147; 120 when all tiles were single CTAs'.)
// STU_B200_TILE_N=128 and 256 force either, STU_B200_TILE_CTAS=1 and 2 the last form or the others; with any of them no K is cut.
enum { TILE_NARROW, TILE_WIDE, TILE_SINGLE };
static const char* tile_n_asked() {
  static const char* env = getenv("STU_B200_TILE_N");
  return env;
}
static const char* tile_ctas_asked() {
  static const char* env = getenv("STU_B200_TILE_CTAS");
  return env;
}
static int tile_form(long long rows, long long cols, bool dual, bool single_built, long long* cost = nullptr) {
  const char *env_n = tile_n_asked(), *env_c = tile_ctas_asked();
  const long long pairs = device_pairs(), sms = device_sm_count(), rows2 = (rows + 2 * BM - 1) / (2 * BM);
  const auto waves = [](long long tiles, long long at_a_time) { return (tiles + at_a_time - 1) / at_a_time; };
  const long long wide = 174 * waves(rows2 * ((cols + 255) / 256), pairs);
  const long long narrow = 100 * waves(rows2 * ((cols + 127) / 128), pairs);
  const long long single_waves = waves((rows + BM - 1) / BM * ((cols + 255) / 256), sms), single = 215 * single_waves;
  int form = dual || wide < narrow ? TILE_WIDE : TILE_NARROW;
  if (cost) *cost = std::min(wide, std::min(narrow, single));
  if (env_n && !dual) form = atoi(env_n) == 128 ? TILE_NARROW : TILE_WIDE;
  if (!single_built || (env_c && atoi(env_c) == 2)) return form;
  if (env_c && atoi(env_c) == 1) return TILE_SINGLE;
  if (rows <= BM && single_waves > 1) return form;   // weights from HBM bound either (128 x 50257 x 1024 27.4 and 29.9 us)
  return single < (form == TILE_WIDE ? wide : narrow) ? TILE_SINGLE : form;
}

// What the tiles of a plain product of this many rows and columns take, in hundredths of a wave of the narrow ones.
extern "C" long long stu_linear_tile_cost(int M, int N) {
  long long cost = 0;
  if (M > 0 && N > 0) tile_form(M, N, false, true, &cost);
  return cost;
}

// Plain and residual products that leave pairs idle for long: the tiles that do not fill a wave (all of them where there are fewer than pairs) are
// 256 x 256 whatever the rows, their K is cut into parts of the same length, and split_sum_kernel adds the parts up.  A pair working alone on
// K = 49152 takes 200 us, so what counts is long K: us, as tile_form has it and split, single calls on operands from HBM, 24000 x 1024 x 49152 (6 of
// 376 tiles in the last wave) 1750 -> 1566, 8192 x 768 x 24576 264 -> 204, 1180 x 1024 x 24576 94 -> 62, 251 x 2048 x 98304 322 -> 106, 74 x 512 x 24576 82 -> 24,
// 16384 x 1536 x 6144 213 -> 200, 4096 x 1536 x 6144 74 -> 64, 333 x 1536 x 6144 29 -> 24.  (That the whole tiles add up the same parts costs, back to back,
// 24000 x 1024 x 8192 269 -> 274, 16384 x 1536 x 6144 201.5 -> 203.4, 19851 x 512 x 3072 50.0 -> 53.4.)  The parts' way through L2 and the second launch cost what short K
// gains: 834 x 768 x 3072 in 4 parts 20.5 -> 21.5, 1337 x 1024 x 2048 in 3 12.6 -> 17.6, 8192 x 1536 x 6144 in 3 106 -> 107.  The line, in us: a k-block
// of 64 takes 0.31 in a wide tile (0.18 in a narrow one; 0.27 and 0.155 where few SMs work), a wave of parts 1 more, each part 0.05 (256 KB
// written and read), the second launch 4; 105 products of 65 to 24000 rows, K = 512 to 98304: 0.97 (noise, not split) to 4.0 times as fast.
static SplitK split_plan(long long M, long long N, long long K) {
  SplitK s = {0, 1, nullptr};
  if (M <= 64 || K < 1024 || tile_n_asked() || tile_ctas_asked()) return s;   // token steps' kernels, never worth it, or another form asked for
  const long long tiles = (M + 255) / 256 * ((N + 255) / 256), pairs = device_pairs(), kb = (K + BK - 1) / BK, rest = tiles % pairs;
  if (rest == 0) return s;
  long long cost = 0;
  tile_form(M, N, false, true, &cost);
  double best = 0.95 * 0.0018 * cost * kb;
  for (long long parts = 2; parts <= std::min(kb, 32ll) && rest * parts <= 5 * pairs; parts++) {   // up to 97 MB of parts
    const double us = tiles / pairs * kb * 0.31 + (rest * parts + pairs - 1) / pairs * ((kb + parts - 1) / parts * 0.31 + 1) + 4 + rest * parts * 0.05;
    if (us < best) best = us, s.parts = (int)parts;
  }
  s.whole = (int)(tiles - rest);
  return s;
}
// fp32 values that stu_linear_split wants for its parts; 0: nothing is split.
extern "C" long long stu_linear_workspace_elems(int M, int N, int K, int epilogue, int dtype) {
  if (dtype != STU_BF16 || (epilogue & ~(STU_FLAG_OVERLAP | STU_FLAG_EARLY_TRIGGER)) > EPI_RESID || M <= 0 || N <= 0 || K <= 0) return 0;
  const SplitK s = split_plan(M, N, K);
  return s.parts > 1 ? ((M + 255ll) / 256 * ((N + 255ll) / 256) - s.whole) * s.parts * SPLIT_TILE : 0;
}

int gemm_tc_dispatch(const void* A, long long lda, const void* B, long long ldb, const void* B2, int M, int N,
                     int K, int epi, int causal, const EpiArgsAny& epa, cudaStream_t st, float* workspace, long long workspace_elems) {
  CUtensorMap ma, mb, mb2;
  EpiArgs<bf16> ep = epa.as<bf16>();
  int rc;
  if (epi == EPI_HIST) {
    // swap operands: rows = channels (the weight), columns = tokens, so that each epilogue thread owns
    // one channel row of the history and writes whole 16-byte runs per parity
    const bool wide = tile_form(N, M, false, false) == TILE_WIDE;
    if ((rc = make_map(&ma, B, N, K, ldb)) != STU_OK) return rc;
    if ((rc = make_map(&mb, A, M, K, lda, wide ? 128 : 64)) != STU_OK) return rc;
    ep.ldy = N;  // channel count
    if (wide) return launch_tc<EPI_HIST_T, 6, 256>(ma, mb, mb, N, M, K, /*m_fast=*/1, 0, ep, device_status_word(), st);
    return launch_tc<EPI_HIST_T, 4, 128>(ma, mb, mb, N, M, K, /*m_fast=*/1, 0, ep, device_status_word(), st);
  }
  if (workspace && !causal && !ep.kpos && !ep.peer && (epi == EPI_STORE || epi == EPI_RESID)) {
    const long long want = stu_linear_workspace_elems(M, N, K, epi, STU_BF16);
    if (want > 0 && want <= workspace_elems) {
      SplitK split = split_plan(M, N, K);
      split.partials = workspace;
      if ((rc = make_map(&ma, A, M, K, lda)) != STU_OK) return rc;
      if ((rc = make_map(&mb, B, N, K, ldb, 128)) != STU_OK) return rc;
      if (epi == EPI_STORE) return launch_tc<EPI_STORE, 6, 256, 2, true>(ma, mb, mb, M, N, K, 0, 0, ep, device_status_word(), st, split);
      return launch_tc<EPI_RESID, 6, 256, 2, true>(ma, mb, mb, M, N, K, 0, 0, ep, device_status_word(), st, split);
    }
  }
  const bool dual = epi == EPI_GELU_MUL;
  const int form = tile_form(M, dual ? 2ll * N : N, dual, epi != EPI_BLOCKCOL);
  if ((rc = make_map(&ma, A, M, K, lda)) != STU_OK) return rc;
  if ((rc = make_map(&mb, B, N, K, ldb, form == TILE_NARROW ? 64 : form == TILE_SINGLE && !dual ? 256 : 128)) != STU_OK) return rc;
  mb2 = mb;
  if (dual && (rc = make_map(&mb2, B2, N, K, ldb)) != STU_OK) return rc;
  if (form == TILE_SINGLE) {
    switch (epi) {
      case EPI_STORE: return launch_tc<EPI_STORE, 4, 256, 1>(ma, mb, mb2, M, N, K, 0, causal, ep, device_status_word(), st);
      case EPI_RESID: return launch_tc<EPI_RESID, 4, 256, 1>(ma, mb, mb2, M, N, K, 0, causal, ep, device_status_word(), st);
      case EPI_GELU_MUL: return launch_tc<EPI_GELU_MUL, 4, 128, 1>(ma, mb, mb2, M, N, K, 0, 0, ep, device_status_word(), st);
    }
  }
  if (form == TILE_WIDE && !dual) {
    switch (epi) {
      case EPI_STORE: return launch_tc<EPI_STORE, 6, 256>(ma, mb, mb2, M, N, K, 0, causal, ep, device_status_word(), st);
      case EPI_RESID: return launch_tc<EPI_RESID, 6, 256>(ma, mb, mb2, M, N, K, 0, causal, ep, device_status_word(), st);
      case EPI_BLOCKCOL:
        return launch_tc<EPI_BLOCKCOL, 6, 256>(ma, mb, mb2, M, N, K, 0, causal, ep, device_status_word(), st);
    }
  }
  switch (epi) {
    case EPI_STORE: return launch_tc<EPI_STORE, 4, 128>(ma, mb, mb2, M, N, K, 0, causal, ep, device_status_word(), st);
    case EPI_RESID: return launch_tc<EPI_RESID, 4, 128>(ma, mb, mb2, M, N, K, 0, causal, ep, device_status_word(), st);
    case EPI_GELU_MUL: return launch_tc<EPI_GELU_MUL, 6, 128>(ma, mb, mb2, M, N, K, 0, 0, ep, device_status_word(), st);
    case EPI_BLOCKCOL: return launch_tc<EPI_BLOCKCOL, 4, 128>(ma, mb, mb2, M, N, K, 0, causal, ep, device_status_word(), st);
  }
  return STU_ERR_UNSUPPORTED;
}

// Token-step linears of 9..64 rows on the tensor cores with swapped operands (skinny_umma_kernel).
// STU_B200_DISABLE_UMMA_SKINNY=1 keeps them on the mma.sync weight-streaming kernels.
bool skinny_umma_takes(int M, int N, int K, int epi, bool norm, bool peer) {
  static const bool off = getenv("STU_B200_DISABLE_UMMA_SKINNY") != nullptr;
  if (off || peer || norm) return false;
  if (epi != EPI_STORE && epi != EPI_RESID && epi != EPI_GELU_MUL) return false;
  // up to 8 rows the 8-feature mma.sync kernel is faster (8 x 4096 x 1024 gate/up 6.0 against 6.3 us, down 4.5 against
  // 5.8 us); from 9 rows on this kernel is (16 rows: gate/up 6144 x 1536 14.2 -> 10.1 us, down 12.6 -> 7.9 us)
  static const int min_rows = getenv("STU_B200_UMMA_MIN_ROWS") ? atoi(getenv("STU_B200_UMMA_MIN_ROWS")) : 9;   // tuning aid
  return M >= min_rows && M <= 64 && K % 8 == 0 && K >= 128 && N >= 64;
}

int skinny_umma_dispatch(const void* A, long long lda, const void* B, long long ldb, const void* B2, int M, int N,
                         int K, int epi, const EpiArgs<bf16>& ep, int pdl, cudaStream_t st) {
  const bool dual = epi == EPI_GELU_MUL;
  CUtensorMap mw, mw2, mx;
  int rc = make_map(&mw, B, N, K, ldb, dual ? 64 : 128);
  if (rc != STU_OK) return rc;
  rc = make_map(&mw2, dual ? B2 : B, N, K, ldb, dual ? 64 : 128);
  if (rc != STU_OK) return rc;
  rc = make_map(&mx, A, M, K, lda, M <= 16 ? 16 : (M <= 32 ? 32 : 64));
  if (rc != STU_OK) return rc;
  // split K over a cluster until there is about one CTA per SM, every CTA keeping at least two 64-element blocks
  // (six for the step from 8 to 16 CTAs per cluster: down 1536 x 6144 at 32 rows 8.4 -> 7.8 us, the 16 x 1024 x 49152
  // contraction of the distilled-LDS features 31.9 -> 21.8 us, but c_proj 1536 x 1536 5.2 -> 5.6 us)
  const int tiles = (N + (dual ? 64 : 128) - 1) / (dual ? 64 : 128), num_kb = (K + BK - 1) / BK;
  const int sms = device_sm_count();
  int ks = 1;
  while (ks < 16 && tiles * ks < sms - sms / 8 && num_kb / (2 * ks) >= (ks >= 8 ? 6 : 2)) ks *= 2;
  if (const char* kv = getenv("STU_B200_UMMA_KS")) ks = atoi(kv);   // tuning aid
  const int early = (pdl & STU_FLAG_OVERLAP) ? 1 : 0;
  int* status = device_status_word();
  switch (epi) {
    case EPI_STORE: return launch_skinny_umma_split<EPI_STORE>(ks, mw, mw2, mx, M, N, K, ep, early, status, st);
    case EPI_RESID: return launch_skinny_umma_split<EPI_RESID>(ks, mw, mw2, mx, M, N, K, ep, early, status, st);
    case EPI_GELU_MUL:
      return launch_skinny_umma_split<EPI_GELU_MUL>(ks, mw, mw2, mx, M, N, K, ep, early, status, st);
  }
  return STU_ERR_UNSUPPORTED;
}
