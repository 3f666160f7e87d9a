// The cached token step of the full STU variant for many channels and long histories, its sums on the 5th-generation tensor cores (what
// full_step_kernel of stu_full_step.cu computes; flash_stu/modules/stu.py:100-118 for the new position t = 2 sn + p).
//
// A CTA owns 64 channels of one sequence: 128 history rows (channel, parity) are the A operand, 64 entries of each per stage, and
// the reversed taps, K even ones and K odd ones of the same entries, the B operand; both come by TMA straight into the swizzled operand layout.  Of
// the 128 x 2K sums a row needs the even taps (its parity is the position's) or the odd ones: the other half is work that costs nothing
// beside the history's bytes.  What the cache holds past the position is set to zero in shared memory ahead of the last stage's instructions.
//
// Bound: HBM, the history once, behind a chain of 7 us back to back (position, first copies, last instructions, outputs) and of 14 behind a kernel that
// it was not launched beside (8 x 1024, history from HBM, at 3000 22.5 us, at 6000 30.7: 49 MB more in 8.2).  full_step_kernel is bound by its load
// units: 16-byte loads of 64-byte pieces of rows, for the taps as many as for the history, 1.9 us for every 256 entries whether they come from
// L1 or from HBM.  us, that one and this one, 24 filters, history from L2: 8 x 1024 channels at position 1000 10.7 and 9.5, at 3000 19.6 and 14.1, at
// 8000 40 and 31; 16 x 1024 at 2000 28.2 and 15.7.  ops.full_decode_step_tc5_pays says where that one stays the faster.
//
// Roles: warp 0 TMA, warp 1 tcgen05.mma, warps 2..5 the RMSNorm of the new input, the last stage's zeros, and the outputs.  Every wait is bounded: on
// expiry the CTA raises status 9, lets issued copies land (bounded), frees its tensor memory and returns.
#include <cuda.h>

#include "common.cuh"
#include "tma.cuh"

int device_sm_count();   // gemm_tc.cu
int operand_map(CUtensorMap* map, const void* base, long long rows, long long cols, long long ld, int box_rows);   // gemm_tc.cu

namespace {

constexpr int CH = 64, BK = 64, THREADS = 192, MAX_K = 32;
constexpr int A_BYTES = 2 * CH * BK * 2;
constexpr int STATUS_WAIT = 9;
constexpr int MAX_STAGES = 6;

struct Ctl {
  uint64_t full[MAX_STAGES], empty[MAX_STAGES], last, fixed, acc_full;   // last: the position's stage, whose rows end in it
 
  uint32_t tmem_slot;
  int abort_flag, issued, consumed, t;
  float part[4], xn[CH], tap0[MAX_K];
};
__host__ __device__ constexpr int stage_bytes(int K8) { return A_BYTES + 2 * K8 * BK * 2; }
constexpr size_t smem_bytes(int K8, int stages) { return 1024 + (size_t)stages * stage_bytes(K8) + sizeof(Ctl); }

__device__ __forceinline__ uint64_t desc_sw128(uint32_t saddr) {   // K-major, 128-byte swizzle
  return (uint64_t)((saddr >> 4) & 0x3FFF) | (uint64_t)1 << 16 | (uint64_t)(1024 >> 4) << 32 | (uint64_t)1 << 46 | (uint64_t)2 << 61;
}
__device__ __forceinline__ void load_2d(void* dst, const CUtensorMap* map, uint64_t* bar, int x, int y) {
  asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
               ::"r"(tma::smem_u32(dst)), "l"(map), "r"(tma::smem_u32(bar)), "r"(x), "r"(y)
               : "memory");
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
__device__ __forceinline__ void outputs_sync() { asm volatile("bar.sync 1, 128;" ::: "memory"); }   // warps 2..5

__global__ void __launch_bounds__(THREADS, 2)
    full_step_umma_kernel(const __grid_constant__ CUtensorMap tmH, const __grid_constant__ CUtensorMap tmT, const bf16* __restrict__ x,
                          long long x_rstride, const bf16* __restrict__ nw, float eps, bf16* __restrict__ hist, const bf16* __restrict__ taps,
                          int* __restrict__ pos, bf16* __restrict__ U, int B, int d, int K, int Lh, int limit, int both,
                          int stages, int* __restrict__ status, int drop_first_stage, unsigned long long wait_ns) {
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  const int K8 = (K + 7) & ~7, stage = stage_bytes(K8);
  Ctl* ctl = reinterpret_cast<Ctl*>(smem + stages * stage);
  volatile int* abort_flag = &ctl->abort_flag;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int per_seq = d / CH, b = blockIdx.x / per_seq, i0 = (blockIdx.x - b * per_seq) * CH;
  if (tid == 0) {
    for (int s = 0; s < stages; s++) {
      tma::mbar_init(&ctl->full[s], 1);
      tma::mbar_init(&ctl->empty[s], 1);
    }
    tma::mbar_init(&ctl->last, 1);
    tma::mbar_init(&ctl->fixed, 128);
    tma::mbar_init(&ctl->acc_full, 1);
    ctl->abort_flag = 0;
    ctl->issued = ctl->consumed = 0;
    tma::fence_barrier_init();
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 64;" ::"r"(tma::smem_u32(&ctl->tmem_slot)));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::);
  }
  // behind everything in front of this launch (see PdlTrigger, epilogue.cuh)
  pdl_wait();
  pdl_trigger();
  if (tid == 0) ctl->t = *(volatile int*)pos;
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = ctl->tmem_slot;
  const int t = ctl->t;
  const bool live = t >= 0 && t < limit;
  const int p = t & 1, sn = t >> 1;
  const int cnt_same = sn, cnt_other = p ? sn + 1 : sn;   // entries of the rows of the position's parity and of the other one
  const int n = live ? (cnt_other + BK - 1) / BK : 0;   // stages
  if (warp == 0) {
    // ---------------- TMA
    const bool leader = elect_one();
    const int oE = Lh - 1 - sn, oQ = Lh - cnt_other;   // tap of entry 0 in the reversed rows; its rest mod 8 picks the table
    int it = 0, s = 0;
    uint32_t ph = 1;
    for (; it < n; it++) {
      if (!tma::warp_wait_bounded(&ctl->empty[s], ph, abort_flag, wait_ns)) break;
      if (leader) {
        unsigned char* a = smem + s * stage;
        uint64_t* bar = it == n - 1 ? &ctl->last : &ctl->full[s];
        tma::mbar_expect_tx(bar, A_BYTES + 2 * K * BK * 2);
        const int e0 = it * BK;
        if (!(drop_first_stage && it == 0)) {   // (a test: these copies are never issued)
          load_2d(a, &tmH, bar, e0, (b * d + i0) * 2);
          load_2d(a + A_BYTES, &tmT, bar, (oE & ~7) + e0, (oE & 7) * 2 * K);
          load_2d(a + A_BYTES + K8 * BK * 2, &tmT, bar, (oQ & ~7) + e0, (oQ & 7) * 2 * K + K);
        }
      }
      __syncwarp();
      if (++s == stages) s = 0, ph ^= 1u;
    }
    if (leader) ctl->issued = it;
  } else if (warp == 1) {
    // ---------------- MMA
    const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(2 * K8 >> 3) << 17) | ((uint32_t)(2 * CH >> 4) << 24);
    const bool leader = elect_one();
    const uint64_t da0 = desc_sw128(tma::smem_u32(smem)), db0 = desc_sw128(tma::smem_u32(smem) + A_BYTES);
    int it = 0, s = 0;
    uint32_t ph = 0;
    for (; it < n; it++) {
      const bool end = it == n - 1;
      if (!tma::warp_wait_bounded(end ? &ctl->fixed : &ctl->full[s], end ? 0u : ph, abort_flag, wait_ns)) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      if (leader) {
        const uint64_t da = da0 + (uint64_t)(s * (stage >> 4)), db = db0 + (uint64_t)(s * (stage >> 4));
#pragma unroll
        for (int kk = 0; kk < BK / 16; kk++) umma(tmem, da + 2 * kk, db + 2 * kk, idesc, it || kk ? 1u : 0u);
        umma_commit(&ctl->empty[s]);
        if (end) umma_commit(&ctl->acc_full);
      }
      __syncwarp();
      if (++s == stages) s = 0, ph ^= 1u;
    }
    if (leader) ctl->consumed = it;
    if (lane == 0 && live) {   // beside the last instructions: the last CTA that has read the position moves it on
      __threadfence();
      if (atomicAdd(&pos[1], 1) == (int)gridDim.x - 1) {
        pos[1] = 0;
        for (int i = 0; i < B; i++)
          if (pos[2 * i] >= 0 && pos[2 * i] < 2 * Lh) pos[2 * i] += 1;
      }
    }
    __syncwarp();
  } else if (!live) {
    if (tid == 64 && blockIdx.x == 0 && status) atomicExch(status, 2);
  } else {
    // ---------------- the new input, normalised as the norm kernel would have stored it
    const int e = tid - 64, quarter = warp & 3, row = quarter * 32 + lane;   // tensor memory: a warp reads the 32 rows of its number mod 4
    const bf16* xr = x + (size_t)b * x_rstride;
    float r = 1.f, mine = 0.f, w = 0.f;
    if (e < CH) {
      mine = Elem<bf16>::to_f(xr[i0 + e]);
      if (nw) w = Elem<bf16>::to_f(nw[i0 + e]);
    } else if (e - CH < K) {
      ctl->tap0[e - CH] = Elem<bf16>::to_f(taps[(size_t)(e - CH) * (Lh + 8) + Lh - 1]);
    }
    if (nw) {
      float ss = 0.f;
      for (int v = e; v * 8 < d; v += 128) {
        float f[8];
        load_vec(xr + v * 8, f);
#pragma unroll
        for (int j = 0; j < 8; j++) ss += f[j] * f[j];
      }
      ss = warp_sum(ss);
      if (lane == 0) ctl->part[warp - 2] = ss;
      outputs_sync();
      r = rsqrtf((ctl->part[0] + ctl->part[1] + ctl->part[2] + ctl->part[3]) / (float)d + eps);
    }
    if (e < CH) {
      const bf16 xn = __float2bfloat16_rn(nw ? mine * r * w : mine);
      ctl->xn[e] = Elem<bf16>::to_f(xn);
      hist[((size_t)((size_t)b * d + i0 + e) * 2 + p) * Lh + sn] = xn;
    }
    outputs_sync();
    bool ok = true;
    if (n > 0) {   // row e of the last stage from its first entry past the position on (this launch's new input among them)
      const int s = (n - 1) % stages, keep = ((e & 1) == p ? cnt_same : cnt_other) - (n - 1) * BK;
      ok = tma::warp_wait_bounded(&ctl->last, 0, abort_flag, wait_ns);
      if (ok) {
        unsigned char* arow = smem + s * stage + e * 128;
        for (int j = keep >> 3; j < 8; j++) {   // 0 <= keep <= 64
          uint4* w = reinterpret_cast<uint4*>(arow + ((j ^ (e & 7)) << 4));
          const int left = keep - j * 8;
          if (left <= 0) {
            *w = make_uint4(0, 0, 0, 0);
          } else {
            uint32_t* q = reinterpret_cast<uint32_t*>(w);
#pragma unroll
            for (int i = 0; i < 4; i++) q[i] = left >= 2 * i + 2 ? q[i] : (left == 2 * i + 1 ? q[i] & 0xffffu : 0u);
          }
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        tma::mbar_arrive(&ctl->fixed);
      }
    }
    // ---------------- the sums: row = channel * 2 + parity; even taps in columns 0.., odd ones in K8..
    const bool same = (row & 1) == p;
    float v[MAX_K];
#pragma unroll
    for (int k = 0; k < MAX_K; k++) v[k] = 0.f;
    if (n > 0) {
      ok = ok && tma::warp_wait_bounded(&ctl->acc_full, 0, abort_flag, wait_ns);
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      uint32_t ev[32], od[32];
      const uint32_t addr = tmem + ((uint32_t)(quarter * 32) << 16);
      tmem_ld32(addr, ev);
      tmem_ld32(addr + K8, od);
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
#pragma unroll
      for (int k = 0; k < MAX_K; k++) v[k] = __uint_as_float(same ? ev[k] : od[k]);
    }
    const auto put = [&](int k, float mine) {
      const float his = __shfl_xor_sync(0xffffffffu, mine, 1);
      const float E = round_to<bf16>((same ? mine : his) + ctl->xn[row >> 1] * ctl->tap0[k]), Q = round_to<bf16>(same ? his : mine);
      bf16* u = U + ((size_t)b * (both ? 2 : 1) * K + k) * d + i0 + (row >> 1);
      if (!(row & 1)) *u = __float2bfloat16_rn(E + Q);
      else if (both) u[(size_t)K * d] = __float2bfloat16_rn(E - Q);
    };
#pragma unroll
    for (int k = 0; k < MAX_K; k++)
      if (k < K && ok) put(k, v[k]);
  }
  __syncwarp();
  __syncthreads();
  if (*abort_flag) {
    if (tid == 0) {
      if (status) atomicExch(status, STATUS_WAIT);
      const uint64_t start = tma::global_ns();
      for (int it = ctl->consumed; it < ctl->issued; it++)
        for (uint32_t w = 0; w < (1u << 22); ++w) {
          if (it == n - 1 ? tma::mbar_try_wait(&ctl->last, 0) : tma::mbar_try_wait(&ctl->full[it % stages], (uint32_t)(it / stages) & 1u)) break;
          if ((w & 255u) == 255u && tma::global_ns() - start > wait_ns) break;
        }
    }
    __syncthreads();
  }
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 64;" ::"r"(tmem));
  }
}

}  // namespace

// stu_full_decode_step (same arguments, same results but for the order of the sums) for d a multiple of 64.
extern "C" int stu_full_decode_step_tc5(const void* x, long long x_rstride, const void* norm_w, float eps, void* hist, const void* taps8, int* pos,
                                        void* U, int B, int d, int K, int Lh, int limit, int both_signs, int* status, int dtype, void* stream) {
  if (!x || !hist || !taps8 || !pos || !U) return STU_ERR_NULL;
  if (B <= 0 || d <= 0 || K <= 0 || Lh <= 0 || limit <= 0 || limit > 2 * Lh) return STU_ERR_SHAPE;
  if (dtype != STU_BF16) return STU_ERR_DTYPE;
  if (K > MAX_K || d % CH || (long long)B * d > (1ll << 29)) return STU_ERR_UNSUPPORTED;
  if (Lh % 8 || !aligned16(hist) || !aligned16(taps8)) return STU_ERR_ALIGN;
  if (norm_w && (x_rstride % 8 || !aligned16(x))) return STU_ERR_ALIGN;
  CUtensorMap h, tp;
  int rc = operand_map(&h, hist, 2ll * B * d, Lh, Lh, 2 * CH);
  if (rc == STU_OK) rc = operand_map(&tp, taps8, 16ll * K, Lh + 8, Lh + 8, K);
  if (rc != STU_OK) return rc;
  static SmemLimit lim;
  cudaError_t e = allow_smem((const void*)full_step_umma_kernel, smem_bytes(MAX_K, MAX_STAGES), lim);
  if (e != cudaSuccess) return (int)e;
  // Four stages where the grid fills more than one CTA per SM, so that two fit (16 x 1024 at position 2000 15.0 us, with six 21.9); six below that (the
  // layer step of 8 x 1024 at 3000 in a chain 51.4 with four, 50.4 with six; two and three, beside which the next kernel's CTAs fit and take the
  // bandwidth early, 57).
  const int tiles = B * (d / CH), stages = tiles > device_sm_count() ? 4 : MAX_STAGES;
  e = launch_maybe_overlapped(full_step_umma_kernel, dim3(tiles), dim3(THREADS), smem_bytes((K + 7) & ~7, stages), (cudaStream_t)stream, true, h, tp,
                              (const bf16*)x, x_rstride, (const bf16*)norm_w, eps, (bf16*)hist, (const bf16*)taps8, pos, (bf16*)U, B, d, K, Lh, limit,
                              both_signs, stages, status, (int)take_dropped_stage(), wait_bound_ns());
  if (e != cudaSuccess) return (int)e;
  STU_CHECK_LAUNCH();
  return STU_OK;
}
