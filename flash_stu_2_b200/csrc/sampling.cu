// Next-token selection from the last-position logits (reference flash_stu/model.py:268-299):
//   z = clamp(logits / temperature, -1e4, 1e4)  (division rounded to the logits dtype)
//   top-k: keep z >= k-th largest (ties kept); top-p: sort kept descending (ties by index), drop an
//   entry when the probability mass ranked before it exceeds top_p; then argmax (greedy) or a draw.
// The reference draws with torch.multinomial; here one uniform u in [0,1) per sequence selects the
// first kept vocabulary index whose running sum of exp(z - max) (vocabulary order) exceeds u * total,
// which is reproducible across devices.
// One CTA of 1024 threads per sequence.  The scaled logits of the row are computed once, in the argmax pass, and kept
// as order-preserving 32-bit keys in shared memory when the vocabulary fits (<= 52 k entries), so the later passes
// neither re-read the logits nor repeat the division.  top-k uses a 4-pass radix select over those keys;
// when top-k is given the (<= 1024) survivors are gathered, sorted by rank in shared memory and the
// nucleus cut and the draw are made on that list, otherwise the draw scans the whole vocabulary.
#include <cooperative_groups.h>
#include <stdlib.h>

#include "common.cuh"

namespace cg = cooperative_groups;

constexpr int SP_T = 1024;
constexpr int SP_CAND = 1024;

__device__ __forceinline__ uint32_t ord_key(float f) {
  uint32_t u = __float_as_uint(f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float key_value(uint32_t k) {   // inverse of ord_key
  return __uint_as_float((k & 0x80000000u) ? (k & 0x7fffffffu) : ~k);
}
constexpr int SP_CACHE_MAX = 50 * 1024 + 512;   // vocabulary entries whose keys fit beside the other shared arrays
constexpr int SP_SUBH = 16;                     // radix histograms per CTA (one per pair of warps), two 16-bit bins per word

template <typename T> __device__ __forceinline__ float scaled_logit(const T* row, int i, float temperature) {
  float z = round_to<T>(__fdiv_rn(Elem<T>::to_f(row[i]), temperature));
  return fminf(fmaxf(z, -1e4f), 1e4f);
}

// Sorts the n <= SP_T first entries, whole CTA; before(a, b): a ranks before b.  Up to SP_RANK of them every entry counts those
// in front of it (the reads are broadcasts): two barriers, where a bitonic network of 128 entries has 28.  With the running sums
// read eight ahead, and two radix passes in place of four for bf16 logits: one row of 50257 entries, top-k 100, top-p 0.9, 27 ->
// 17 us.  The counts grow with the square: from there on the network, whose padding ranks last.  Counts and network, us, one row
// of 50257, top-p 0.9: top-k 257 77 and 80, 400 87 and 84, 513 98 and 95, 700 110 and 100, 1000 134 and 107; without a nucleus
// (one sort) 400 75 and 76, 700 96 and 91.
constexpr int SP_RANK = 512;
template <typename F> __device__ __forceinline__ void sort_candidates(float* s_val, int* s_idx, int n, F before) {
  const int tid = threadIdx.x;
  if (n > SP_RANK) {
    int width = 2 * SP_RANK;   // (a power of two)
    while (width < n) width <<= 1;
    if (tid >= n && tid < width) {
      s_val[tid] = -INFINITY;
      s_idx[tid] = 0x7fffffff;
    }
    __syncthreads();
    for (int k = 2; k <= width; k <<= 1)
      for (int j = k >> 1; j > 0; j >>= 1) {
        const int other = tid ^ j;
        if (other > tid && other < width) {
          const float va = s_val[tid], vb = s_val[other];
          const int ia = s_idx[tid], ib = s_idx[other];
          if (((tid & k) == 0) != before(va, ia, vb, ib)) {
            s_val[tid] = vb;
            s_val[other] = va;
            s_idx[tid] = ib;
            s_idx[other] = ia;
          }
        }
        __syncthreads();
      }
    return;
  }
  float v = 0.f;
  int id = 0, rank = 0;
  if (tid < n) {
    v = s_val[tid];
    id = s_idx[tid];
#pragma unroll 8
    for (int r = 0; r < n; r++) {
      const float vr = s_val[r];
      const int ir = s_idx[r];
      rank += before(vr, ir, v, id);   // (a strict order of distinct entries)
    }
  }
  __syncthreads();
  if (tid < n) {
    s_val[rank] = v;
    s_idx[rank] = id;
  }
  __syncthreads();
}

// Nucleus cut and draw among the C <= SP_CAND survivors of top-k (any order), whole CTA of SP_T threads.  The sums run
// over the entries one by one (fp32, deterministic) in one thread; the exponentials and quotients that they add up are
// computed beside each other first.
__device__ __forceinline__ void draw_from_candidates(float* s_val, int* s_idx, int C, float zmax, float top_p, float u,
                                                     long long* out) {
  __shared__ float s_exp[SP_CAND];
  __shared__ float s_tot;
  __shared__ int s_keep;
  const int tid = threadIdx.x;
  if (tid == 0) s_keep = C;
  __syncthreads();
  if (top_p > 0.f && top_p < 1.f) {
    sort_candidates(s_val, s_idx, C, [](float va, int ia, float vb, int ib) { return va > vb || (va == vb && ia < ib); });
    if (tid < C) s_exp[tid] = __expf(s_val[tid] - zmax);
    __syncthreads();
    if (tid == 0) {
      float tot = 0.f;
#pragma unroll 8
      for (int r = 0; r < C; r++) tot += s_exp[r];
      s_tot = tot;
    }
    __syncthreads();
    if (tid < C) s_exp[tid] = s_exp[tid] / s_tot;
    __syncthreads();
    if (tid == 0) {
      float cum = 0.f;
      int keep = 0;
      for (int r0 = 0; keep == r0 && r0 < C; r0 += 8) {   // eight at a time: their reads are not behind the sums
        float e[8];
#pragma unroll
        for (int j = 0; j < 8; j++) e[j] = r0 + j < C ? s_exp[r0 + j] : 0.f;
#pragma unroll
        for (int j = 0; j < 8; j++)
          if (keep == r0 + j && r0 + j < C && !(r0 + j > 0 && cum > top_p)) {
            keep = r0 + j + 1;
            cum += e[j];
          }
      }
      s_keep = keep;
    }
    __syncthreads();
  }
  const int keep = s_keep;
  // the kept entries by index ascending, for the running sum in vocabulary order
  sort_candidates(s_val, s_idx, keep, [](float, int ia, float, int ib) { return ia < ib; });
  if (tid < keep) s_exp[tid] = __expf(s_val[tid] - zmax);
  __syncthreads();
  if (tid == 0) {
    float tot = 0.f;
#pragma unroll 8
    for (int r = 0; r < keep; r++) tot += s_exp[r];
    const float target = u * tot;
    float cum = 0.f;
    int chosen = keep - 1;
    bool found = false;
    for (int r0 = 0; !found && r0 < keep; r0 += 8) {
      float e[8];
#pragma unroll
      for (int j = 0; j < 8; j++) e[j] = r0 + j < keep ? s_exp[r0 + j] : 0.f;
#pragma unroll
      for (int j = 0; j < 8; j++)
        if (!found && r0 + j < keep) {
          cum += e[j];
          if (cum > target) {
            chosen = r0 + j;
            found = true;
          }
        }
    }
    *out = s_idx[chosen];
  }
}

// The bin (of 256 counts) that holds the need-th largest key, by one warp: 8 bins per lane, suffix sums across the lanes.
// The owner lane moves need and prefix on.
__device__ __forceinline__ void pick_bin(const unsigned* hist, unsigned need, unsigned prefix, int shift, unsigned* s_need,
                                         unsigned* s_prefix) {
  const int lane = threadIdx.x & 31;
  unsigned t = 0;
#pragma unroll
  for (int j = 0; j < 8; j++) t += hist[8 * lane + j];
  unsigned S = t;   // bins of this lane and of all higher lanes
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned n = __shfl_down_sync(0xffffffffu, S, o);
    if (lane + o < 32) S += n;
  }
  const unsigned reach = __ballot_sync(0xffffffffu, S >= need);
  const int owner = reach ? 31 - __clz(reach) : 0;   // highest lane whose suffix reaches the need (else bin 0)
  if (lane == owner) {
    unsigned cum = S - t;
    int bin = 8 * lane + 7;
    for (; bin > 8 * lane; bin--) {
      if (cum + hist[bin] >= need) break;
      cum += hist[bin];
    }
    // (the lowest bin of the owner's range takes what is left, as bin 0 does in a sequential scan)
    *s_need = need - cum;
    *s_prefix = prefix | ((unsigned)bin << shift);
  }
}

// One row by one CTA.  cache: the scaled keys of the row are kept in s_key [V]; full: the filters over the whole
// vocabulary are available (the row would fit there).
template <typename T>
__device__ void sample_row(int b, uint32_t* s_key, const T* __restrict__ logits, long long ld, int V, float temperature,
                           int top_k, float top_p, int do_sample, const float* __restrict__ uniforms,
                           long long* __restrict__ out, long long out_stride, int* __restrict__ status, int cache,
                           int full, int variant) {
  __shared__ unsigned int s_sub[SP_SUBH][128];
  __shared__ float s_val[SP_CAND];
  __shared__ int s_idx[SP_CAND];
  __shared__ unsigned int s_hist[256];
  __shared__ float s_red[32];
  __shared__ int s_redi[32];
  __shared__ unsigned int s_prefix, s_need, s_count;
  __shared__ int s_choice;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const T* row = logits + (size_t)b * ld;
  auto key_at = [&](int i) { return cache ? s_key[i] : ord_key(scaled_logit(row, i, temperature)); };

  // ---- argmax (lowest index among ties); also the fallback result
  float best = -INFINITY;
  int besti = V;
  int saw_nan = 0;
  for (int i = tid; i < V; i += SP_T) {
    float z = scaled_logit(row, i, temperature);
    saw_nan |= isnan(Elem<T>::to_f(row[i])) ? 1 : 0;   // (the clamp inside scaled_logit would hide it)
    if (cache) s_key[i] = ord_key(z);
    if (z > best || (z == best && i < besti)) { best = z; besti = i; }
  }
  saw_nan = __syncthreads_or(saw_nan);
  // scaled logit of entry i for the later passes
  auto zval = [&](int i) { return cache ? key_value(s_key[i]) : scaled_logit(row, i, temperature); };
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    float ob = __shfl_xor_sync(0xffffffffu, best, o);
    int oi = __shfl_xor_sync(0xffffffffu, besti, o);
    if (ob > best || (ob == best && oi < besti)) { best = ob; besti = oi; }
  }
  if (lane == 0) { s_red[warp] = best; s_redi[warp] = besti; }
  __syncthreads();
  if (warp == 0) {
    best = s_red[lane]; besti = s_redi[lane];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      float ob = __shfl_xor_sync(0xffffffffu, best, o);
      int oi = __shfl_xor_sync(0xffffffffu, besti, o);
      if (ob > best || (ob == best && oi < besti)) { best = ob; besti = oi; }
    }
    if (lane == 0) { s_red[0] = best; s_redi[0] = besti; }
  }
  __syncthreads();
  const float zmax = s_red[0];
  const int imax = s_redi[0];
  if (!do_sample) {
    if (tid == 0) out[(size_t)b * out_stride] = imax < V ? imax : 0;
    return;
  }
  const float u = uniforms[b];
  if (saw_nan) {
    // a NaN logit makes the reference's softmax NaN everywhere and it falls back to a uniformly random token
    // (flash_stu/model.py:293-296); here the row's uniform picks it
    if (tid == 0) out[(size_t)b * out_stride] = min(V - 1, (int)(u * (float)V));
    return;
  }

  // ---- radix select: key of the need-th largest scaled logit (4 passes of 8 bits); all threads call it
  auto select_kth = [&](unsigned need_total) -> unsigned {
    if (tid == 0) { s_prefix = 0; s_need = need_total; }
    for (int pass = 0; pass < 4; pass++) {
      const int shift = 24 - 8 * pass;
      if (tid < 256) s_hist[tid] = 0;
      for (int i = tid; i < SP_SUBH * 128; i += SP_T) (&s_sub[0][0])[i] = 0;
      __syncthreads();
      const unsigned prefix = s_prefix;
      const unsigned mask = pass == 0 ? 0u : (0xffffffffu << (shift + 8));
      // logits share their sign and exponent bytes, so almost every key of a pass lands in one or two bins.  Each
      // pair of warps counts into a histogram of its own (16-bit counters, two per word: a row has fewer than
      // 65536 entries), which are summed afterwards; with one shared histogram the 32 warps queue on one counter.
      unsigned int* sub = s_sub[warp >> 1];
      for (int base = 0; base < V; base += SP_T) {
        const int i = base + tid;
        unsigned bin = 0xffffffffu;
        if (i < V) {
          const unsigned key = key_at(i);
          if ((key & mask) == prefix) bin = (key >> shift) & 255u;
        }
        if (variant == 0) {
          const unsigned peers = __match_any_sync(0xffffffffu, bin);
          if (bin != 0xffffffffu && lane == __ffs(peers) - 1) atomicAdd(&s_hist[bin], (unsigned)__popc(peers));
        } else if (variant == 1) {
          if (bin != 0xffffffffu) atomicAdd(&sub[bin >> 1], 1u << (16 * (bin & 1)));
        } else {
          const unsigned peers = __match_any_sync(0xffffffffu, bin);
          if (bin != 0xffffffffu && lane == __ffs(peers) - 1)
            atomicAdd(&sub[bin >> 1], (unsigned)__popc(peers) << (16 * (bin & 1)));
        }
      }
      __syncthreads();
      if (variant != 0 && tid < 256) {
        unsigned c = 0;
#pragma unroll
        for (int h = 0; h < SP_SUBH; h++) c += (s_sub[h][tid >> 1] >> (16 * (tid & 1))) & 0xffffu;
        s_hist[tid] = c;
      }
      __syncthreads();
      if (warp == 0) pick_bin(s_hist, s_need, prefix, shift, &s_need, &s_prefix);
      __syncthreads();
    }
    const unsigned r = s_prefix;
    __syncthreads();
    return r;
  };
  unsigned floor_from_list = 0;   // set when the candidate list overflows (ties): the full-vocabulary path takes over
  if (top_k > 0 && top_k <= SP_CAND && top_k < V) {
    const unsigned kth_key = select_kth((unsigned)top_k);
    // ---- gather survivors (key >= kth_key)
    if (tid == 0) s_count = 0;
    __syncthreads();
    for (int i = tid; i < V; i += SP_T) {
      float z = zval(i);
      if (ord_key(z) >= kth_key) {
        unsigned slot = atomicAdd(&s_count, 1u);
        if (slot < SP_CAND) { s_val[slot] = z; s_idx[slot] = i; }
      }
    }
    __syncthreads();
    const int C = (int)s_count;
    if (C > SP_CAND && !full) {  // more ties than the candidate list holds: report and return the argmax
      if (tid == 0) {
        if (status) atomicExch(status, 4);
        out[(size_t)b * out_stride] = imax;
      }
      return;
    }
    if (C > SP_CAND) {
      floor_from_list = kth_key;   // (a key of a finite logit is never 0)
    } else {
      draw_from_candidates(s_val, s_idx, C, zmax, top_p, u, out + (size_t)b * out_stride);
      return;
    }   // candidate list
  }
  // ---- full-vocabulary filters: nucleus without top-k, or a top-k wider than the candidate list (with or without a
  //      nucleus cut inside it).  Needs the row's keys in shared memory.
  const bool big_k = (top_k > SP_CAND && top_k < V) || floor_from_list != 0;
  const bool nucleus = top_p > 0.f && top_p < 1.f;
  unsigned keep_key = 0;          // entries with a key above this are kept ...
  unsigned tie_key = 0xffffffffu; // ... and, of the entries equal to tie_key, the first tie_keep in vocabulary order
  unsigned tie_keep = 0;
  bool filtered = false;
  if (big_k || nucleus) {
    if (!full) {   // the vocabulary does not fit in shared memory
      if (tid == 0) {
        if (status) atomicExch(status, nucleus ? 5 : 4);
        out[(size_t)b * out_stride] = imax;
      }
      return;
    }
    filtered = true;
    unsigned floor_key = 0;   // top-k: keys below this are out (ties with the k-th are kept, as in the reference)
    if (big_k) floor_key = floor_from_list ? floor_from_list : select_kth((unsigned)top_k);
    if (!nucleus) {
      keep_key = floor_key > 0 ? floor_key - 1 : 0;
      if (floor_key == 0) filtered = false;
    } else {
      // Probability mass as 40-bit fixed point of exp(z - zmax): integer sums do not depend on the order of the
      // additions, so the cut is reproducible.  Sorted by (value descending, index ascending) an entry is kept while
      // the mass ranked before it is <= top_p * total (flash_stu/model.py:284-291): find the key v* at which the mass
      // from the top first exceeds that bound (4 passes of 8 bits over mass histograms); keys above v* are kept, of
      // the entries equal to v* the first floor((bound - mass above) / mass of one) + 1 in vocabulary order.
      unsigned long long* mh = reinterpret_cast<unsigned long long*>(&s_sub[0][0]);   // [4][256]
      auto mass_of = [&](unsigned key) {
        return (unsigned long long)(__expf(key_value(key) - zmax) * 1099511627776.f);   // 2^40
      };
      __shared__ unsigned long long s_total, s_bound, s_above;
      if (tid == 0) s_total = 0;
      __syncthreads();
      {
        unsigned long long part = 0;
        for (int i = tid; i < V; i += SP_T)
          {
            const unsigned key = key_at(i);
            if (key >= floor_key) part += mass_of(key);
          }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
        if (lane == 0) atomicAdd(&s_total, part);
      }
      __syncthreads();
      if (tid == 0) {
        s_bound = (unsigned long long)((double)top_p * (double)s_total);
        s_above = 0;
        s_prefix = 0;
      }
      __syncthreads();
      for (int pass = 0; pass < 4; pass++) {
        const int shift = 24 - 8 * pass;
        for (int i = tid; i < 4 * 256; i += SP_T) mh[i] = 0;
        __syncthreads();
        const unsigned prefix = s_prefix;
        const unsigned mask = pass == 0 ? 0u : (0xffffffffu << (shift + 8));
        unsigned long long* sub = mh + (warp >> 3) * 256;
        for (int i = tid; i < V; i += SP_T) {
          const unsigned key = key_at(i);
          if (key >= floor_key && (key & mask) == prefix) atomicAdd(&sub[(key >> shift) & 255u], mass_of(key));
        }
        __syncthreads();
        if (tid == 0) {
          // from the top bin down: the first bin whose mass pushes the running sum over the bound holds v*
          unsigned long long cum = s_above;
          const unsigned long long bound = s_bound;
          int bin = 255;
          for (; bin > 0; bin--) {
            const unsigned long long hb = mh[bin] + mh[256 + bin] + mh[512 + bin] + mh[768 + bin];
            if (cum + hb > bound) break;
            cum += hb;
          }
          s_above = cum;
          s_prefix = prefix | ((unsigned)bin << shift);
        }
        __syncthreads();
      }
      tie_key = s_prefix;
      if (tie_key < floor_key) tie_key = floor_key;   // the bound was never exceeded: everything above the floor stays
      keep_key = tie_key;
      const unsigned long long one = mass_of(tie_key);
      const unsigned long long room = s_bound >= s_above ? s_bound - s_above : 0;
      tie_keep = one ? (unsigned)min((unsigned long long)V, room / one + 1ull) : (unsigned)V;
      __syncthreads();
    }
  }
  // entry i survives the filters: above the cut, or one of the first tie_keep entries equal to the cut key (their
  // rank among the ties in vocabulary order is supplied by the caller)
  auto kept = [&](unsigned key, unsigned tie_rank) {
    return !filtered || key > keep_key || (key == tie_key && tie_rank < tie_keep);
  };

  // ---- plain temperature sampling over the whole vocabulary: chunked running sum in index order
  const int chunk = (V + SP_T - 1) / SP_T;
  const int lo = tid * chunk, hi = min(V, lo + chunk);
  // ties with the cut key before this thread's chunk (vocabulary order): exclusive scan of the per-thread counts
  unsigned tie_base = 0;
  if (filtered && tie_key != 0xffffffffu) {
    unsigned mine = 0;
    for (int i = lo; i < hi; i++) mine += (key_at(i) == tie_key);
    unsigned incl_t = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned n = __shfl_up_sync(0xffffffffu, incl_t, o);
      if (lane >= o) incl_t += n;
    }
    if (lane == 31) s_redi[warp] = (int)incl_t;
    __syncthreads();
    unsigned before = 0;
    for (int w = 0; w < warp; w++) before += (unsigned)s_redi[w];
    tie_base = before + incl_t - mine;
    __syncthreads();
  }
  float part = 0.f;
  {
    unsigned tr = tie_base;
    for (int i = lo; i < hi; i++) {
      const unsigned key = filtered ? key_at(i) : 0u;
      if (kept(key, tr)) part += __expf(zval(i) - zmax);
      if (filtered && key == tie_key) tr++;
    }
  }
  // block exclusive scan of the 1024 partial sums
  float incl = part;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    float n = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += n;
  }
  if (lane == 31) s_red[warp] = incl;
  __syncthreads();
  if (warp == 0) {
    float w = s_red[lane], wi = w;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      float n = __shfl_up_sync(0xffffffffu, wi, o);
      if (lane >= o) wi += n;
    }
    s_red[lane] = wi - w;  // exclusive prefix of warp totals
    if (lane == 31) s_hist[0] = __float_as_uint(wi);
  }
  if (tid == 0) s_choice = 0x7fffffff;
  __syncthreads();
  const float tot = __uint_as_float(s_hist[0]);
  const float target = u * tot;
  const float excl = s_red[warp] + incl - part;
  if (lo < hi && part > 0.f && excl <= target && target < excl + part) {
    float cum = excl;
    int choice = -1;
    unsigned tr = tie_base;
    for (int i = lo; i < hi; i++) {
      const unsigned key = filtered ? key_at(i) : 0u;
      if (kept(key, tr)) {
        choice = i;   // the last kept entry of the chunk takes what rounding leaves over
        cum += __expf(zval(i) - zmax);
        if (cum > target) break;
      }
      if (filtered && key == tie_key) tr++;
    }
    if (choice >= 0) atomicMin(&s_choice, choice);
  }
  __syncthreads();
  if (tid == 0) out[(size_t)b * out_stride] = (s_choice == 0x7fffffff) ? imax : s_choice;
}

template <typename T>
__global__ void __launch_bounds__(SP_T) sample_kernel(const T* __restrict__ logits, long long ld, int V,
                                                      float temperature, int top_k, float top_p, int do_sample,
                                                      const float* __restrict__ uniforms, long long* __restrict__ out,
                                                      long long out_stride, int* __restrict__ status, int cache,
                                                      int variant) {
  extern __shared__ uint32_t s_key[];   // [V] when cache
  sample_row<T>(blockIdx.x, s_key, logits, ld, V, temperature, top_k, top_p, do_sample, uniforms, out, out_stride, status,
                cache, cache, variant);
}

// Greedy selection and top-k of at most SPC_TOPK, one cluster of 8 CTAs per row.  Bound: latency; one CTA walked the row
// in 49 steps per pass, six passes.  Here a thread holds at most 8 entries, in registers, read once; the four radix
// passes add the CTAs' histograms through distributed shared memory, every CTA for itself, and the survivors meet in
// CTA 0, which cuts and draws as sample_row does: the same token.  More survivors than the list holds (ties): CTA 0
// runs sample_row.  The figures stand at the rule in stu_sample.
constexpr int SPC = 8, SPC_PER = 8, SPC_TOPK = 256;
constexpr int SPC_MAX_V = SPC * SP_T * SPC_PER;
template <typename T>
__global__ void __cluster_dims__(SPC, 1, 1) __launch_bounds__(SP_T, 2)
    sample_cluster_kernel(const T* __restrict__ logits, long long ld, int V, float temperature, int top_k, float top_p,
                          int do_sample, const float* __restrict__ uniforms, long long* __restrict__ out,
                          long long out_stride, int* __restrict__ status, int full) {
  __shared__ unsigned s_sub[8][256];    // one histogram per four warps
  __shared__ unsigned s_own[4][256];    // this CTA's counts of each pass (read by the others: never reused)
  __shared__ unsigned s_hist[256];
  __shared__ float s_val[SP_CAND];
  __shared__ int s_idx[SP_CAND];
  __shared__ float s_red[32];
  __shared__ int s_redi[32];
  __shared__ float s_best;
  __shared__ int s_besti, s_nan;
  __shared__ unsigned s_prefix, s_need, s_count;
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = (int)cluster.block_rank(), b = blockIdx.x / SPC;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const T* row = logits + (size_t)b * ld;
  const int slice = (V + SPC - 1) / SPC, lo = rank * slice, hi = min(V, lo + slice);

  float best = -INFINITY;
  int besti = V, saw_nan = 0;
  float raw[SPC_PER];
#pragma unroll
  for (int j = 0; j < SPC_PER; j++) {
    const int i = lo + tid + j * SP_T;
    raw[j] = i < hi ? Elem<T>::to_f(row[i]) : 0.f;
  }
  unsigned key[SPC_PER];   // 0 past the end: no finite value has that key
#pragma unroll
  for (int j = 0; j < SPC_PER; j++) {
    const int i = lo + tid + j * SP_T;
    key[j] = 0;
    if (i < hi) {
      saw_nan |= isnan(raw[j]) ? 1 : 0;
      const float z = fminf(fmaxf(round_to<T>(__fdiv_rn(raw[j], temperature)), -1e4f), 1e4f);   // scaled_logit
      key[j] = ord_key(z);
      if (z > best || (z == best && i < besti)) { best = z; besti = i; }
    }
  }
  saw_nan = __syncthreads_or(saw_nan);
  auto better = [](float a, int ai, float c, int ci) { return c > a || (c == a && ci < ai); };
  auto warp_best = [&]() {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float ob = __shfl_xor_sync(0xffffffffu, best, o);
      const int oi = __shfl_xor_sync(0xffffffffu, besti, o);
      if (better(best, besti, ob, oi)) { best = ob; besti = oi; }
    }
  };
  warp_best();
  if (lane == 0) { s_red[warp] = best; s_redi[warp] = besti; }
  __syncthreads();
  if (warp == 0) {
    best = s_red[lane]; besti = s_redi[lane];
    warp_best();
    if (lane == 0) { s_best = best; s_besti = besti; s_nan = saw_nan; s_count = 0; s_prefix = 0; s_need = (unsigned)top_k; }
  }
  cluster.sync();
  float zmax = -INFINITY;
  int imax = V, nan_row = 0;
#pragma unroll
  for (int r = 0; r < SPC; r++) {
    const float ob = *cluster.map_shared_rank(&s_best, r);
    const int oi = *cluster.map_shared_rank(&s_besti, r);
    nan_row |= *cluster.map_shared_rank(&s_nan, r);
    if (better(zmax, imax, ob, oi)) { zmax = ob; imax = oi; }
  }
  if (!do_sample || nan_row) {   // the same in every CTA of the cluster
    if (rank == 0 && tid == 0)   // a NaN logit: the row's uniform picks the token, see sample_row
      out[(size_t)b * out_stride] = !do_sample ? (imax < V ? imax : 0) : min(V - 1, (int)(uniforms[b] * (float)V));
    cluster.sync();              // the others' values have been read
    return;
  }
  for (int pass = 0; pass < 4; pass++) {
    const int shift = 24 - 8 * pass;
    for (int i = tid; i < 8 * 256; i += SP_T) (&s_sub[0][0])[i] = 0;
    __syncthreads();
    const unsigned prefix = s_prefix, need = s_need;
    const unsigned mask = pass == 0 ? 0u : (0xffffffffu << (shift + 8));
#pragma unroll
    for (int j = 0; j < SPC_PER; j++) {
      const unsigned bin = key[j] != 0 && (key[j] & mask) == prefix ? (key[j] >> shift) & 255u : 0xffffffffu;
      if (__all_sync(0xffffffffu, bin == 0xffffffffu)) continue;
      const unsigned peers = __match_any_sync(0xffffffffu, bin);   // almost all keys share a bin: one atomic per warp
      if (bin != 0xffffffffu && lane == __ffs(peers) - 1) atomicAdd(&s_sub[warp >> 2][bin], (unsigned)__popc(peers));
    }
    __syncthreads();
    if (tid < 256) {
      unsigned c = 0;
#pragma unroll
      for (int h = 0; h < 8; h++) c += s_sub[h][tid];
      s_own[pass][tid] = c;
    }
    cluster.sync();
    if (tid < 256) {
      unsigned c = 0;
#pragma unroll
      for (int r = 0; r < SPC; r++) c += *cluster.map_shared_rank(&s_own[pass][tid], r);
      s_hist[tid] = c;
    }
    __syncthreads();
    if (warp == 0) pick_bin(s_hist, need, prefix, shift, &s_need, &s_prefix);
    __syncthreads();
    // bf16 logits: the keys of a bin of the upper 16 bits are all the same, but in the two that hold the clamp's bounds, which
    // are no bf16 values.  What counts below is key >= prefix.
    if (sizeof(T) == 2 && pass == 1) {
      const unsigned top = s_prefix >> 16;
      if (top != ord_key(1e4f) >> 16 && top != ord_key(-1e4f) >> 16) break;   // the same in every CTA
    }
  }
  const unsigned kth_key = s_prefix;
#pragma unroll
  for (int j = 0; j < SPC_PER; j++)
    if (key[j] != 0 && key[j] >= kth_key) {
      const unsigned slot = atomicAdd(&s_count, 1u);
      if (slot < SP_CAND) {
        s_val[slot] = key_value(key[j]);
        s_idx[slot] = lo + tid + j * SP_T;
      }
    }
  cluster.sync();
  unsigned C = 0;
  if (rank == 0) {
#pragma unroll
    for (int r = 0; r < SPC; r++) {
      const unsigned n = *cluster.map_shared_rank(&s_count, r);
      if (r > 0 && C + n <= SP_CAND && tid < (int)n) {
        s_val[C + tid] = cluster.map_shared_rank(s_val, r)[tid];
        s_idx[C + tid] = cluster.map_shared_rank(s_idx, r)[tid];
      }
      C += n;
    }
  }
  cluster.sync();   // the lists have been read
  if (rank != 0) return;
  if (C <= SP_CAND)
    draw_from_candidates(s_val, s_idx, (int)C, zmax, top_p, uniforms[b], out + (size_t)b * out_stride);
  else
    sample_row<T>(b, nullptr, logits, ld, V, temperature, top_k, top_p, do_sample, uniforms, out, out_stride, status, 0, full, 0);
}

// logits [B, V] (row stride ld); uniforms [B] fp32 on the device (read only when do_sample);
// out[b * out_stride] receives the token id (int64).  top_k <= 0 and top_p outside (0,1) disable the filters.
extern "C" int stu_sample(const void* logits, long long ld, int B, int V, float temperature, int top_k, float top_p,
                          int do_sample, const float* uniforms, long long* out, long long out_stride, int* status,
                          int dtype, void* stream) {
  if (!logits || !out) return STU_ERR_NULL;
  if (do_sample && !uniforms) return STU_ERR_NULL;
  if (B <= 0 || V <= 0 || !(temperature > 0.f)) return STU_ERR_SHAPE;
  if (top_k > SP_CAND && top_k < V && V > SP_CACHE_MAX) return STU_ERR_UNSUPPORTED;   // needs the row in shared memory
  cudaStream_t st = (cudaStream_t)stream;
  // greedy selection makes one pass only: nothing to keep
  const int cache = (do_sample && V <= SP_CACHE_MAX) ? 1 : 0;
  static const int variant = getenv("STU_SAMPLE_VARIANT") ? atoi(getenv("STU_SAMPLE_VARIANT")) : 2;
  // A cluster per row where the row fits the cluster's registers and is long enough to pay for the cluster's barriers.  37
  // rows are resident (two CTAs per SM), so its time grows with the rows and doubles past 37, while one CTA per row takes
  // the same time for any number up to 148; past SPC_TOPK the survivors of a bf16 row may well exceed the list.
  // Measured, us, one CTA and a cluster per row:
  //   greedy     1 row: 16384 entries 5.9 and 7.1, 50257 13.0 and 7.7; 32 rows: 50257 13.0 and 13.2, 65536 15.8 and 13.4;
  //              64 rows: 65536 15.9 and 24.0
  //   top-k 40   1 row: 4096 entries 20.4 and 20.1, 16384 32.8 and 21.2; 32 rows: 4096 21.4 and 27.9, 16384 34.3 and 29.2;
  //              64 rows: 16384 34.8 and 53.8, 50257 74.0 and 57.9
  const bool wins = !do_sample ? B <= 32 && V >= 24576 + 768 * B
                               : top_k > 0 && top_k <= SPC_TOPK && (B <= 32 ? V >= 6144 + 256 * B : B <= 64 && V >= 36864);
  if (wins && V <= SPC_MAX_V) {
    const int full = V <= SP_CACHE_MAX;
    if (dtype == STU_F32)
      sample_cluster_kernel<float><<<B * SPC, SP_T, 0, st>>>((const float*)logits, ld, V, temperature, top_k, top_p,
                                                             do_sample, uniforms, out, out_stride, status, full);
    else if (dtype == STU_BF16)
      sample_cluster_kernel<bf16><<<B * SPC, SP_T, 0, st>>>((const bf16*)logits, ld, V, temperature, top_k, top_p,
                                                            do_sample, uniforms, out, out_stride, status, full);
    else
      return STU_ERR_DTYPE;
    STU_CHECK_LAUNCH();
    return STU_OK;
  }
  const size_t smem = cache ? (size_t)V * sizeof(uint32_t) : 0;
  if (dtype == STU_F32) {
    if (cache) {
      cudaError_t e = cudaFuncSetAttribute(sample_kernel<float>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           SP_CACHE_MAX * (int)sizeof(uint32_t));
      if (e != cudaSuccess) return (int)e;
    }
    sample_kernel<float><<<B, SP_T, smem, st>>>((const float*)logits, ld, V, temperature, top_k, top_p, do_sample,
                                                uniforms, out, out_stride, status, cache, (V < 65536) ? variant : 0);
  } else if (dtype == STU_BF16) {
    if (cache) {
      cudaError_t e = cudaFuncSetAttribute(sample_kernel<bf16>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           SP_CACHE_MAX * (int)sizeof(uint32_t));
      if (e != cudaSuccess) return (int)e;
    }
    sample_kernel<bf16><<<B, SP_T, smem, st>>>((const bf16*)logits, ld, V, temperature, top_k, top_p, do_sample,
                                               uniforms, out, out_stride, status, cache, (V < 65536) ? variant : 0);
  } else {
    return STU_ERR_DTYPE;
  }
  STU_CHECK_LAUNCH();
  return STU_OK;
}
