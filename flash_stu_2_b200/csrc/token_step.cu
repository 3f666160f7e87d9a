// One token step of a stack of layers (approx STU and sliding-window attention layers in any order, each with its
// MLP), optionally from the token ids to the logits, as ONE persistent kernel for at most 8 sequences at one common
// position.  Reference semantics: flash_stu/layers/stu_layer.py:78-97, flash_stu/layers/attention_layer.py:50-66,
// flash_stu/modules/{stu,attention,swiglu}.py and flash_stu/model.py:150-205 for the new position only.
//
// Bound: HBM (every weight once per step: 1.8 GB = 283 us for the 24-layer 1536-wide bf16 model) against the chain of
// dependent products (96 of them).  Launched kernel by kernel the chain wins: a dependent launch costs 2.5 us before
// its first byte, and at most one kernel ahead can fetch its weights.  Here one CTA per SM runs the whole chain, and the weight
// stream does not stop between two products: a producer warp walks the
// weight rows of ALL products of ALL layers in order and brings them by bulk copies (one piece of d values each; pieces
// below 2 KB are bound by the copy engine's request rate) into a ring of row slots (up to 180 KB per SM, 26 MB over
// the chip), however far the arithmetic is.
//
//   product      a CTA owns N / 148 consecutive output features (no tile granularity), its 8 consumer warps split K
//   activations  the input rows of a product (at most 8 x max(d, I)) are read from L2 into shared memory, times the norm
//                weight when the product is behind a norm, and feed every feature of the CTA
//   hand-over    results travel as tagged words (below), which the readers poll: a grid barrier waits for the stores, for an
//                atomic to arrive and for another read to see it before the first row can be read.  That model, 1 sequence: 771
//                -> 683 us a step; 12 fp32 layers of 512, 2 sequences: 352 -> 311.  Barriers are left where the words would be
//                read by everybody in bulk: the attention's partial sums, and rows of many bytes (TAGGED_X_BYTES).  With them and
//                rows in fours, 5 to 8 sequences of 1536, 6 layers, take 281 to 296 us (339 to 359 with words alone, 268 to 278
//                with barriers alone, in less code)
//   STU          a CTA's channels are projected, appended to the history and combined with their tap sums in place;
//                the tap sums over the cached history need nothing of this step and are taken ahead of the wait
//   attention    (sequence, head, key range) items over the CTAs; the ranges are merged by the readers
//
// bf16: mma.sync m16n8k16, weights as the 16-row operand (gate/up: 8 gate and the 8 up rows of the same features),
// sequences as the 8 columns.  fp32: FMAs.  All product code exists once (a stage switch picks operands and epilogue):
// written out per product it outgrew the instruction cache (that model, 1 sequence: 1.25 ms a step where this form took 0.75).
// Every wait is bounded: on expiry the status word is raised, outstanding copies are let land and every CTA returns.  The
// caches, positions and outputs are then undefined, and the workspace is marked: launches on it return at once with the
// same status (their barriers would start from a counter that was left half way) until it is zeroed.
#include "../../include/stu_b200.h"   // the descriptors
#include "common.cuh"
#include "tma.cuh"

int device_sm_count();   // gemm_tc.cu

namespace {

constexpr int NW = 8, CONS = NW * 32, THREADS = CONS + 32;   // consumer warps, and the producer warp
constexpr int MAXL = STU_STEP_MAX_LAYERS;
constexpr int TILES = 6;                      // tiles whose partial sums wait in shared memory
constexpr int STEP_SMEM = 210 * 1024;         // beside 15 KB of static shared memory
constexpr int RED_BYTES = TILES * NW * 128 * 4;
constexpr uint32_t COPY = 4096;                // bytes of one bulk copy at most
constexpr int UNITS = 32;                     // row groups in flight
constexpr int MAX_ROWS = 32;                  // STU channels per CTA
// Rows are handed over as tagged words up to these sizes, by a barrier and as plain values above (every CTA reads all of a product's
// rows: twice the bytes).  us a step, tagged and plain.  The residual stream, 32 KB: 24 KB (bf16, 4 rows of 1536, 6 layers) 233 and
// 239, 32 KB (fp32, 4 rows of 1024, 6 layers) 234 and 243, (bf16, 8 of 1024, 10 layers) 365 and 376, 48 KB (8 of 1536) 299 and 297,
// (fp32, 8 of 768, 10 layers) 455 and 447.  The rows of the down projection, 100 KB for one and two sequences, half of that for
// more: 48 KB (bf16, 4 of 3072, 18 layers) 405 and 417, 96 KB (fp32, 2 of 6144, 8 layers) 207 and 210, (bf16, 4 of 6144, 6 layers)
// 239 and 234, (fp32, 4 of 3072, 10 layers) 312 and 296, 128 KB (fp32, 4 of 4096, 6 layers) 249 and 243, 192 KB (bf16, 8 of 6144) 314
// and 295.
constexpr long long TAGGED_X_BYTES = 32 * 1024, TAGGED_H_BYTES = 100 * 1024;
constexpr int MAX_VECS = 2 * CONS;            // 16-byte vectors of a row of the residual stream at most
static_assert(2 * MAX_VECS * 32 <= TAGGED_X_BYTES, "one or two rows of the residual stream are always handed over as words");

__device__ __forceinline__ void cons_bar() { asm volatile("bar.sync 1, 256;" ::: "memory"); }
__device__ __forceinline__ uint4 ldcg16(const void* p) { return __ldcg(reinterpret_cast<const uint4*>(p)); }
__device__ __forceinline__ uint4 ldnc16(const void* p) {
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "l"(p));
  return v;
}
__device__ __forceinline__ void mma_16816(float* c, uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                          uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void unpack(const uint4& v, float (&o)[8], bf16*) {
  const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
  for (int i = 0; i < 4; i++) {
    o[2 * i] = __uint_as_float(w[i] << 16);
    o[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
  }
}
__device__ __forceinline__ void unpack(const uint4& v, float (&o)[4], float*) {
  o[0] = __uint_as_float(v.x); o[1] = __uint_as_float(v.y); o[2] = __uint_as_float(v.z); o[3] = __uint_as_float(v.w);
}
__device__ __forceinline__ float ldcg_f(const float* p) { return __ldcg(p); }
__device__ __forceinline__ float ldcg_f(const bf16* p) {
  return __uint_as_float((uint32_t)__ldcg(reinterpret_cast<const unsigned short*>(p)) << 16);
}
// Tagged words: a value that one CTA hands to all others, and beside it in the same word the number of the use of its buffer
// that it belongs to.  A reader polls the word itself: neither a fence nor a counter stands between the store and the load
// that finds it.  bf16: 32 bits, the value above 16 bits of tag; fp32: 64 bits, the tag above the value.
// (Every write of a word carries another tag than the write before: see tag_of in the kernel.)
// The elements of a reader's 16-byte load are as wide as the stores: the parts of a vector access are accesses of their own, so only
// a value and a tag of one element come from one store.
template <typename T> struct Tagged;
template <> struct Tagged<bf16> {
  static constexpr int BYTES = 4;
  static __device__ __forceinline__ uint4 load(const char* p) {
    uint4 v;
    asm volatile("ld.relaxed.gpu.global.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
    return v;
  }
  static __device__ __forceinline__ bool has(const uint4& w, uint32_t tag) {
    return (((w.x ^ tag) | (w.y ^ tag) | (w.z ^ tag) | (w.w ^ tag)) & 0xffffu) == 0;
  }
  static __device__ __forceinline__ uint2 values(const uint4& w) {   // eight bytes of plain values
    return make_uint2(__byte_perm(w.x, w.y, 0x7632), __byte_perm(w.z, w.w, 0x7632));
  }
  static __device__ __forceinline__ void put(char* row, int i, bf16 v, uint32_t tag) {
    const uint32_t w = ((uint32_t)__bfloat16_as_ushort(v) << 16) | (tag & 0xffffu);
    asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(row + (size_t)i * 4), "r"(w) : "memory");
  }
};
template <> struct Tagged<float> {
  static constexpr int BYTES = 8;
  static __device__ __forceinline__ uint4 load(const char* p) {
    uint64_t a, b;
    asm volatile("ld.relaxed.gpu.global.v2.u64 {%0,%1}, [%2];" : "=l"(a), "=l"(b) : "l"(p) : "memory");
    return make_uint4((uint32_t)a, (uint32_t)(a >> 32), (uint32_t)b, (uint32_t)(b >> 32));
  }
  static __device__ __forceinline__ bool has(const uint4& w, uint32_t tag) { return w.y == tag && w.w == tag; }
  static __device__ __forceinline__ uint2 values(const uint4& w) { return make_uint2(w.x, w.z); }
  static __device__ __forceinline__ void put(char* row, int i, float v, uint32_t tag) {
    const uint64_t w = ((uint64_t)tag << 32) | __float_as_uint(v);
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(row + (size_t)i * 8), "l"(w) : "memory");
  }
};
__device__ __forceinline__ void unpack8(const uint2& v, float (&o)[4], bf16*) {   // the values of eight bytes
  o[0] = __uint_as_float(v.x << 16); o[1] = __uint_as_float(v.x & 0xffff0000u);
  o[2] = __uint_as_float(v.y << 16); o[3] = __uint_as_float(v.y & 0xffff0000u);
}
__device__ __forceinline__ void unpack8(const uint2& v, float (&o)[2], float*) {
  o[0] = __uint_as_float(v.x); o[1] = __uint_as_float(v.y);
}
__device__ __forceinline__ uint2 pack8(const float (&v)[4], bf16*) {
  const __nv_bfloat162 a = __floats2bfloat162_rn(v[0], v[1]), b = __floats2bfloat162_rn(v[2], v[3]);
  return make_uint2(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&b));
}
__device__ __forceinline__ uint2 pack8(const float (&v)[2], float*) { return make_uint2(__float_as_uint(v[0]), __float_as_uint(v[1])); }
// The sum over the warp of v[lane / (32 / NV)] (NV a power of two <= 32).
template <int NV>
__device__ __forceinline__ float fold(float (&v)[NV], int lane) {
  int off = 16;
#pragma unroll
  for (int n = NV; n > 1; n >>= 1, off >>= 1) {
#pragma unroll
    for (int i = 0; i < n / 2; i++) {
      const bool up = (lane & off) != 0;
      const float send = up ? v[i] : v[i + n / 2], keep = up ? v[i + n / 2] : v[i];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, send, off);
    }
  }
#pragma unroll
  for (int o = 16 / NV; o > 0; o >>= 1) v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
  return v[0];
}

// ---- the stages of the chain, in order: the products and, between c_attn and c_proj, the attention itself
enum { ST_STU, ST_QKV, ST_ATTEND, ST_CPROJ, ST_GATE_UP, ST_DOWN, ST_LM_HEAD };
struct Stage {
  const char *W, *W2;   // W2: the up projection (gate and up rows of a feature go together); W null: no product
  int N, K;
  short kind, layer;
  int pieces;           // pieces of d values of a row
};
struct Range { int r0, r1; };   // this CTA's features of a stage
constexpr int MAX_STAGES = 5 * MAXL + 1;
static_assert(sizeof(Stage) == 32 && sizeof(StuStepLayer) == 128, "the plan is copied in 16-byte pieces");
static_assert(sizeof(StuStepArgs) == 128, "as in the Python binding");

struct Params {
  StuStepArgs a;
  const uint4* plan;   // [nst] stages, [n_layers] layers
  int nst;
  int slots, pitch;    // ring: row slots and their distance in bytes
  int xs_cols;         // columns of the activation rows in shared memory: max(d, I), or less, a multiple of d
  float scale;
  int tagged_x, tagged_h;   // the rows of the residual stream, of the down projection, are handed over as tagged words
  int signature;       // of the sizes that the layout of the workspace follows from
};
__host__ __device__ inline Range share_of(int N, unsigned cta, unsigned ctas) {   // N < 2^24 (checked by the host)
  return {(int)((unsigned)N * cta / ctas), (int)((unsigned)N * (cta + 1) / ctas)};
}
__device__ __forceinline__ void prefetch_l2(const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }

// A unit of the weight stream: the rows of one tile of features (16; gate/up: 8, gate rows first, then up rows) over
// one or several pieces of d values, in consecutive slots of the ring (a row's pieces together; a unit does not wrap, it
// skips to slot 0).  Order: product, tile, piece.
// Two layouts.  Rows of 3 KB and more (bf16): slots 64 bytes past a multiple of 128 apart, which makes the fragment loads
// conflict-free, one piece per unit, one bulk copy per row.  Otherwise slots are packed, so that the rows of a unit are
// one copy (gate/up: two; several pieces: one per row): at 52 ns a copy, single rows of 1 KB would cap the stream at
// 2.9 TB/s; bf16 then pays two-way bank conflicts (fp32 has none), and a tile of few rows takes several pieces at once,
// since a unit is a round of waits and arrivals for every warp.
// fp32: warps that share a pair of rows (a power of two; the teams take the pairs in turn).
__device__ __forceinline__ int team_warps(int rows) { return rows > 8 ? 1 : rows > 4 ? 2 : rows > 2 ? 4 : 8; }
// `in_rows`: pieces of the activation rows that are in shared memory at a time; a unit lies inside them.
__host__ __device__ inline int unit_pieces(int rows, int pieces, int slots, bool packed, int in_rows) {
  int p = pieces < in_rows ? pieces : in_rows;
  if (p > slots / (3 * rows)) p = slots / (3 * rows);
  if (!packed || p < 1) p = 1;
  while (in_rows % p) p--;
  return p;
}
// Slots that a unit of n leaves unused in front of itself, from `head` to the end of the ring, because it does not wrap;
// they count as its own until it is released.  Into an empty ring it goes without them: there they are free, and with
// them a unit of 16 rows would fit no ring of fewer than 31 slots whenever it has to skip.
__host__ __device__ inline int unit_skip(int head, int n, int slots, int used) {
  return head + n > slots && used > 0 ? slots - head : 0;
}
template <typename T, int MM>
__global__ void __launch_bounds__(THREADS, 1) token_step_kernel(const __grid_constant__ Params P) {
  constexpr int V = Elem<T>::VEC;
  extern __shared__ __align__(128) unsigned char sm[];
  const StuStepArgs& a = P.a;
  const int slots = P.slots, pitch_w = P.pitch, nst = P.nst;
  int nst_run = nst;
  const int xs_cols = P.xs_cols;
  const bool packed = pitch_w == a.d * (int)sizeof(T);
  unsigned char* ring = sm;
  float* red = reinterpret_cast<float*>(ring + (((size_t)slots * pitch_w + 127) & ~(size_t)127));
  unsigned char* xs = reinterpret_cast<unsigned char*>(red) + RED_BYTES;   // activation rows
  __shared__ uint4 s_plan[MAX_STAGES * 2 + MAXL * 8];
  __shared__ Range s_range[MAX_STAGES];
  __shared__ const T* s_row[8];   // rows of the first layer (null: an id outside the vocabulary)
  __shared__ uint64_t full_bar[UNITS], empty_bar[UNITS];
  __shared__ float s_part[8][NW], s_scale[8];
  __shared__ float s_hist[MAX_ROWS * 8];
  __shared__ int s_abort, s_go[2];
  __shared__ uint64_t s_start;
  const Stage* tab = reinterpret_cast<const Stage*>(s_plan);
  const StuStepLayer* layers = reinterpret_cast<const StuStepLayer*>(s_plan + nst * 2);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, q = lane & 3;
  const int B = a.B, d = a.d, I = a.I, H = a.H, G = gridDim.x, cta = blockIdx.x;
  const int hd = H > 0 ? d / H : V;
  unsigned char* ws = (unsigned char*)a.workspace;
  int* epoch_word = (int*)ws;
  constexpr int TB = Tagged<T>::BYTES;
  // tagged rows: X_ROWS the residual stream behind a layer, MID_ROWS in front of its MLP, QKV_ROWS, H_ROWS the rows of the
  // down projection (plain values where P.tagged_h is 0); behind them the attention's items: hd sums, the maximum and the
  // denominator
  enum { X_ROWS = 0, MID_ROWS = 8, QKV_ROWS = 16, H_ROWS = 40 };
  auto rows_at = [&](int k) { return (char*)a.workspace + 512 + (size_t)(k * d) * TB; };
  auto att_at = [&]() { return (float*)(rows_at(H_ROWS) + (size_t)8 * I * TB); };
  T* xbuf = (T*)a.x;

  for (int i = tid; i < nst * 2 + a.n_layers * 8; i += THREADS) s_plan[i] = __ldg(P.plan + i);
  if (tid == 0) {
    for (int i = 0; i < UNITS; i++) {
      tma::mbar_init(&full_bar[i], 1);
      tma::mbar_init(&empty_bar[i], NW);
    }
    s_abort = 0;
    s_start = tma::global_ns();
    tma::fence_barrier_init();
  }
  // epoch, whether a launch has given up, and the sizes that the tagged words were last written for
  const int4 control = __ldcg(reinterpret_cast<const int4*>(ws));
  const int epoch = control.x;
  __syncthreads();
  for (int i = tid; i < nst; i += THREADS) s_range[i] = share_of(tab[i].N, blockIdx.x, gridDim.x);
  const int t = __ldcg(layers[0].pos);
  int bad = 0;
  for (int i = tid; i < a.n_layers * B; i += THREADS) {
    const StuStepLayer& L = layers[i / B];
    const int tl = __ldcg(L.pos + 2 * (i % B));
    if (tl != t) bad = 6;
    if (tl < 0 || (L.kind == STU_STEP_STU && tl >= 2 * L.Lh)) bad = 2;
  }
  if (control.y) bad = 12;   // its barrier counter is not to be trusted any more
  const int any2 = __syncthreads_or(bad == 2), any6 = __syncthreads_or(bad == 6), any12 = __syncthreads_or(bad == 12);
  if (any2 || any6 || any12) {   // every CTA sees the same words, none waits for another
    if (tid == 0 && cta == 0 && a.status) atomicExch(a.status, any12 ? 12 : any2 ? 2 : 6);
    return;
  }
  int* counter = (int*)(ws + 128 + 128 * (epoch & 1));   // arrivals at the barriers; 16 words on: CTAs that have started
  int* started = counter + 16;
  if (tid == 0) {
    if (cta == 0) {   // the next launch's (the last one that used them has ended)
      int* next = (int*)(ws + 128 + 128 * ((epoch + 1) & 1));
      next[0] = next[16] = 0;
    }
    asm volatile("red.release.gpu.global.add.s32 [%0], 1;" ::"l"(started) : "memory");   // the control words and positions are read
  }

  if (warp == NW) {
    // ================================================================ producer
    int head = 0, used = 0, slots_of = 0;   // next slot, slots taken, slots of the unit with this lane's index
    unsigned issued = 0, freed = 0;
    bool ok = true;
    for (int st = 0; ok && st < nst; st++) {
      const Stage s = tab[st];
      if (!s.W) continue;
      const bool dual = s.W2 != nullptr;
      const int F = dual ? 8 : 16, r1 = s_range[st].r1;
      for (int f0 = s_range[st].r0; ok && f0 < r1; f0 += F) {
        const int nf = min(F, r1 - f0), rows = dual ? 2 * nf : nf;
        // (a lone warp: every division here would show in the stream's rate, 0.6 us a unit before they were hoisted)
        const int pieces = s.pieces == 1 ? 1 : unit_pieces(rows, s.pieces, slots, packed, P.xs_cols / d);
        for (int k0 = 0, p0 = 0; k0 < s.K; k0 += pieces * d, p0 += pieces) {
          const int np = min(pieces, s.pieces - p0), n = rows * np;
          const bool wrap = head + n > slots;   // (then the consumers go on at slot 0 as well)
          int skip = unit_skip(head, n, slots, used);
          while (ok && (used + skip + n > slots || issued - freed == UNITS)) {
            ok = tma::mbar_wait_bounded(&empty_bar[freed % UNITS], (freed / UNITS) & 1u, &s_abort);
            ok = __all_sync(0xffffffffu, ok);
            used -= __shfl_sync(0xffffffffu, slots_of, freed % UNITS);
            freed++;
            skip = unit_skip(head, n, slots, used);
          }
          if (!ok) break;
          if (wrap) head = 0;
          const uint32_t row_bytes = (uint32_t)min(np * d, s.K - k0) * sizeof(T);
          uint64_t* bar = &full_bar[issued % UNITS];
          if (lane == 0) tma::mbar_expect_tx(bar, row_bytes * rows);
          __syncwarp();
          // whole rows of a packed unit lie back to back: the gate rows (or all) and the up rows are one block each
          // (rows that are no whole number of pieces leave the end of their slots unused: one copy per row)
          const bool whole = packed && np == s.pieces && s.K == s.pieces * d;
          const int blocks = whole ? (dual ? 2 : 1) : rows;
          const uint32_t block = whole ? row_bytes * nf : row_bytes;
          const int cuts = (int)((block + COPY - 1) / COPY);   // copies per block
          for (int i = lane; i < blocks * cuts; i += 32) {
            const int b = whole ? (i >= cuts) : cuts == 1 ? i : i / cuts, r = whole ? b * nf : b;
            const uint32_t off = (uint32_t)(i - b * cuts) * COPY;
            const bool up = dual && r >= nf;
            const char* src = (up ? s.W2 : s.W) + ((size_t)(f0 + (up ? r - nf : r)) * s.K + k0) * sizeof(T);
            tma::bulk_load(ring + (size_t)(head + r * np) * pitch_w + off, src + off, min(COPY, block - off), bar);
          }
          if (lane == (int)(issued % UNITS)) slots_of = skip + n;
          head = head + n;
          used += skip + n;
          issued++;
        }
      }
    }
    {   // what was issued has landed before shared memory is released, whatever the consumers did
      for (unsigned u = issued > UNITS ? issued - UNITS : 0; u < issued; u++) {
        int dummy = 0;
        tma::mbar_wait_bounded(&full_bar[u % UNITS], (u / UNITS) & 1u, &dummy, 20000000ull, 1u << 16);
      }
    }
    __syncthreads();   // pairs with the consumers' last barrier
    return;
  }

  // ================================================================ consumers
  const int par = t & 1, s_pos = t >> 1;   // parity row of the history and index in it
  {   // the norm weights of the whole stack towards L2: read behind the weight stream they would each cost its queue
    for (int n = cta * NW + warp; n <= 2 * a.n_layers; n += G * NW) {
      const void* base = n == 2 * a.n_layers ? a.norm_final : ((n & 1) ? layers[n >> 1].norm2 : layers[n >> 1].norm1);
      for (int off = lane * 128; base && off < d * (int)sizeof(T); off += 32 * 128) prefetch_l2((const char*)base + off);
    }
  }
  // ---- attention: key ranges (items) of the CTAs
  const int j_lo = max(0, t - a.window), nkeys = t - j_lo + 1;
  const int S = H > 0 ? max(1, min(min(8, G / (B * H)), (nkeys + 63) / 64)) : 1;
  const int per = (nkeys + S - 1) / S;
  const int LPK = hd / V, KPW = 32 / LPK, sub = lane % LPK, grp = lane / LPK;   // lanes per key, keys per warp and load

  int target = 0;   // arrivals at the barriers so far
  auto arrive = [&]() {
    cons_bar();
    if (tid == 0) asm volatile("red.release.gpu.global.add.s32 [%0], 1;" ::"l"(counter) : "memory");
  };
  // Whether this thread should stop waiting: another has given up, or the launch has taken two seconds (looked at every 64 polls).
  auto give_up = [&](uint32_t polls) -> bool {
    if ((polls & 63u) != 63u) return false;
    if (*(volatile int*)&s_abort) return true;
    if (tma::global_ns() - s_start < 2000000000ull && polls < (1u << 24)) return false;
    *(volatile int*)&s_abort = 1;
    return true;
  };
  auto poll_count = [&](const int* word, int least) {
    for (uint32_t it = 0;; ++it) {
      int v;
      asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(word) : "memory");
      if (v >= least || give_up(it)) return;
    }
  };
  // One answer for the whole CTA, behind a barrier (the producer may raise s_abort at any time)
  unsigned asked = 0;   // (in turn in two words: nobody is two barriers behind)
  auto go_on = [&]() -> bool {
    int* go = s_go + (asked++ & 1u);
    if (tid == 0) *go = *(volatile int*)&s_abort == 0;
    cons_bar();
    return *go;
  };
  auto wait = [&](int arrivals) -> bool {   // `arrivals` more CTAs have arrived than at the last barrier
    target += arrivals;
    if (tid == 0) poll_count(counter, target);
    return go_on();
  };
  // The number of a layer's use of the row buffers.  Consecutive writes of a word differ in it, also in its low 16 bits: the
  // next use is another layer of this launch or a layer of the next one (64 on for the same layer); none is 0 in its low
  // 6 bits, which is what a zeroed word holds.
  auto tag_of = [&](int layer) -> uint32_t { return (uint32_t)epoch * 64u + (uint32_t)layer + 1u; };
  // The values [k0, k0 + len) of the tagged rows m0 .. m0 + RG - 1 (of B) of K, eight bytes of them at a time: use(row - m0, piece,
  // values, extra), extra = more(piece) asked for ahead of the wait.
  constexpr int RG = MM < 4 ? MM : 4;                 // rows on their way at a time (with eight the kernel spills 330 bytes and
                                                      // takes 20 % longer)
  constexpr int VU = MM == 1 ? 4 : MM == 2 ? 2 : 1;   // pieces of a row on their way at a time
  auto take = [&](const char* src, int K, int k0, int len, int m0, uint32_t tag, auto more, auto use) {
    const int nv = len * (int)sizeof(T) / 8, rows = B - m0;
    const char* base = src + ((size_t)m0 * K + k0) * TB;
#pragma unroll 1
    for (int v0 = tid; v0 < nv; v0 += CONS * VU) {
      uint4 w[RG][VU];
      uint2 ex[VU];
#pragma unroll
      for (int u = 0; u < VU; u++) ex[u] = v0 + u * CONS < nv ? more(v0 + u * CONS) : make_uint2(0, 0);
      for (uint32_t it = 0;; ++it) {
        bool all = true;
#pragma unroll
        for (int m = 0; m < RG; m++)
#pragma unroll
          for (int u = 0; u < VU; u++)
            if (m < rows && v0 + u * CONS < nv) w[m][u] = Tagged<T>::load(base + (size_t)m * K * TB + (size_t)(v0 + u * CONS) * 16);
#pragma unroll
        for (int m = 0; m < RG; m++)
#pragma unroll
          for (int u = 0; u < VU; u++)
            if (m < rows && v0 + u * CONS < nv) all = all && Tagged<T>::has(w[m][u], tag);
        if (all || give_up(it)) break;
      }
#pragma unroll
      for (int m = 0; m < RG; m++)
#pragma unroll
        for (int u = 0; u < VU; u++)
          if (m < rows && v0 + u * CONS < nv) use(m, v0 + u * CONS, Tagged<T>::values(w[m][u]), ex[u]);
    }
  };
  // V values at a tagged word, by this thread alone
  auto take_vec = [&](const char* p, uint32_t tag, uint4& out) {
    constexpr int N = V * TB / 16;
    uint4 w[N];
    for (uint32_t it = 0;; ++it) {
      bool all = true;
#pragma unroll
      for (int i = 0; i < N; i++) w[i] = Tagged<T>::load(p + i * 16);
#pragma unroll
      for (int i = 0; i < N; i++) all = all && Tagged<T>::has(w[i], tag);
      if (all || give_up(it)) break;
    }
    const uint2 lo = Tagged<T>::values(w[0]), hi = Tagged<T>::values(w[1]);
    out = make_uint4(lo.x, lo.y, hi.x, hi.y);
  };
  static_assert(V * TB == 32, "two loads of tagged words per vector");
  // A workspace that was last used for other sizes: whatever lies where the tagged words go is cleared first, as in a new one
  if (control.z != P.signature) {
    uint4* words = reinterpret_cast<uint4*>(rows_at(X_ROWS));
    const size_t n = ((size_t)40 * d + (size_t)8 * I) * TB / 16;
    for (size_t i = (size_t)cta * CONS + tid; i < n; i += (size_t)G * CONS) words[i] = make_uint4(0, 0, 0, 0);
    arrive();
  }
  // row m of the input of the first layer
  auto first_row = [&](int m) -> const T* {
    if (!a.ids) return xbuf + (size_t)m * d;
    const long long id = a.ids[(size_t)m * a.ids_stride];
    if (id >= 0 && id < a.V) return (const T*)a.embedding + (size_t)id * d;
    if (cta == 0 && a.status) atomicExch(a.status, 1);
    return nullptr;
  };
  // Results: thread e finishes feature e % n of sequence e / n, n the features of the CTA; of a d-wide product that is at most
  // one per thread, the same one in every layer: it keeps the residual stream there.
  const Range own_r = share_of(d, blockIdx.x, gridDim.x);
  const int c0 = own_r.r0, own = own_r.r1 - c0, my_m = own ? tid / own : 0, my_c = c0 + (own ? tid - my_m * own : 0);
  const bool mine = own && tid < B * own;
  if (tid < B) s_row[tid] = first_row(tid);
  cons_bar();
  float stream = mine && s_row[my_m] ? ldcg_f(s_row[my_m] + my_c) : 0.f;   // this thread's value of the residual stream
  int slot = 0;        // first slot of the next unit
  unsigned unit = 0;   // its index

  // columns [k0, k0 + len) of B plain rows of K values
  auto load_plain = [&](const T* src, int K, int k0, int len, int pitch) {
    const int nv = len / V;
#pragma unroll 1
    for (int v = tid; v < nv; v += CONS) {
      uint4 raw[MM];
#pragma unroll
      for (int m = 0; m < MM; m++) raw[m] = m < B ? ldcg16(src + (size_t)m * K + k0 + v * V) : make_uint4(0, 0, 0, 0);
#pragma unroll
      for (int m = 0; m < MM; m++)
        if (m < B) *reinterpret_cast<uint4*>(xs + m * pitch + v * 16) = raw[m];
    }
  };
  // columns [k0, k0 + len) of the B rows of the down projection
  auto load_h = [&](int layer, int k0, int len, int pitch) {
    if (P.tagged_h) {
#pragma unroll 1
      for (int m0 = 0; m0 < (RG < MM ? B : 1); m0 += RG)
        take(rows_at(H_ROWS), I, k0, len, m0, tag_of(layer), [](int) { return make_uint2(0, 0); },
             [&](int m, int v, const uint2& val, const uint2&) { *reinterpret_cast<uint2*>(xs + (m0 + m) * pitch + v * 8) = val; });
      return;
    }
    load_plain((const T*)rows_at(H_ROWS), I, k0, len, pitch);
  };
  const int down_rows = min(16, own), down_pieces = own > 0 ? unit_pieces(down_rows, (I + d - 1) / d, slots, packed, xs_cols / d) : 1;
  const bool words_x = MM <= 2 || P.tagged_x;   // (one or two rows: at any width, see the host)
  const int items = B * H * S, owners = min(G, items);   // of the attention, and the CTAs that have any
  if (control.z != P.signature && !wait(G)) nst_run = 0;

#pragma unroll 1
  for (int st = 0; st < nst_run; st++) {
    const Stage sg = tab[st];
    const int kind = sg.kind;
    const StuStepLayer& L = layers[min((int)sg.layer, a.n_layers - 1)];
    const bool normed = kind == ST_STU || kind == ST_QKV || kind == ST_GATE_UP || kind == ST_LM_HEAD;
    const int next_kind = st + 1 < nst ? tab[st + 1].kind : -1;

    // ================================================================ ahead of the wait: what needs nothing of this step
    const int r0 = s_range[st].r0, r1 = s_range[st].r1;
    float tap0 = 0.f;
    if (kind == ST_STU) {   // tap sums over the cached history of this CTA's channels
      const T* taps = (const T*)L.taps;
      const int Lh = L.Lh, o = Lh - 1 - s_pos, e8 = o & 7;
#pragma unroll 1
      for (int it0 = warp; it0 < own * B; it0 += 2 * NW) {   // two rows of a warp at a time: one memory round trip
        float sum[2] = {0.f, 0.f};
        const T *hrow[2], *trow[2];
#pragma unroll
        for (int u = 0; u < 2; u++) {
          const int it = min(it0 + u * NW, own * B - 1), m = it / own, c = c0 + it - m * own;
          hrow[u] = (const T*)L.hist + ((size_t)((size_t)m * d + c) * 2 + par) * Lh;
          trow[u] = sizeof(T) == 2 ? taps + (size_t)((size_t)e8 * d + c) * (Lh + 8) + (o - e8) : taps + (size_t)c * Lh + s_pos;
        }
        if constexpr (sizeof(T) == 2) {
#pragma unroll 1
          for (int k = lane * 8; k < s_pos; k += 256) {
            uint4 hr[2], tr[2];
#pragma unroll
            for (int u = 0; u < 2; u++) {
              hr[u] = ldnc16(hrow[u] + k);
              tr[u] = ldnc16(trow[u] + k);
            }
#pragma unroll
            for (int u = 0; u < 2; u++) {
              float hv[8], tv[8];
              unpack(hr[u], hv, (bf16*)nullptr);
              unpack(tr[u], tv, (bf16*)nullptr);
#pragma unroll
              for (int j = 0; j < 8; j++) sum[u] = (k + j < s_pos) ? fmaf(hv[j], tv[j], sum[u]) : sum[u];
            }
          }
        } else {
#pragma unroll 2
          for (int k = lane; k < s_pos; k += 32)
#pragma unroll
            for (int u = 0; u < 2; u++) sum[u] = fmaf((float)hrow[u][k], (float)trow[u][-k], sum[u]);
        }
#pragma unroll
        for (int u = 0; u < 2; u++) {
          sum[u] = warp_sum(sum[u]);
          if (lane == 0 && it0 + u * NW < own * B) s_hist[it0 + u * NW] = sum[u];
        }
      }
      if (mine)
        tap0 = sizeof(T) == 2 ? Elem<T>::to_f(taps[(size_t)my_c * (Lh + 8) + Lh - 1]) : Elem<T>::to_f(taps[(size_t)my_c * Lh]);
    }
    if (kind == ST_QKV) {   // the keys and values that this CTA's items will read, towards L2
      const T *kr = (const T*)L.k_ring, *vr = (const T*)L.v_ring;
      for (int it = cta; it < B * H * S; it += G) {
        const int b = it / (H * S), h = (it / S) % H, k0 = (it % S) * per, k1 = min(nkeys, k0 + per);
        for (int kk = k0 + tid; kk < k1; kk += CONS) {
          const size_t off = ((size_t)b * L.W + (j_lo + kk) % L.W) * d + h * hd;   // (the new token's slot: harmless)
          for (int x = 0; x < hd; x += 128 / (int)sizeof(T)) {
            prefetch_l2(kr + off + x);
            prefetch_l2(vr + off + x);
          }
        }
      }
    }
    if (next_kind == ST_STU) {   // the history and tap rows of the next stage, towards L2
      const StuStepLayer& N = layers[sg.layer + 1];
      const int Lh = N.Lh, o = Lh - 1 - s_pos, e8 = o & 7, bytes = s_pos * (int)sizeof(T);
      if ((long long)own * B * bytes < (1 << 20)) {   // a long history is bandwidth, not latency
        for (int it = warp; it < own * B; it += NW) {
          const int m = it / own, c = c0 + it - m * own;
          const char* hr = (const char*)((const T*)N.hist + ((size_t)((size_t)m * d + c) * 2 + par) * Lh);
          const char* tr = sizeof(T) == 2 ? (const char*)((const T*)N.taps + (size_t)((size_t)e8 * d + c) * (Lh + 8) + (o - e8))
                                          : (const char*)((const T*)N.taps + (size_t)c * Lh);
          for (int off = lane * 128; off < bytes; off += 32 * 128) {
            prefetch_l2(hr + off);
            if (m == 0) prefetch_l2(tr + off);
          }
        }
      }
    }


    if (kind == ST_ATTEND) {
      cons_bar();   // the sums of the product before have been read
      const T *kr = (const T*)L.k_ring, *vr = (const T*)L.v_ring;
      const int W = L.W;
      const float inv_cap = a.softcap > 0.f ? 1.f / a.softcap : 0.f;
#pragma unroll 1
      for (int it = cta; it < items; it += G) {
        const int b = it / (H * S), h = (it / S) % H, sp = it % S;
        const char* cur = rows_at(QKV_ROWS + 3 * b) + h * hd * TB;   // query, key and value of the new token
        const uint32_t tag = tag_of(sg.layer);
        const int k0 = sp * per, k1 = min(nkeys, k0 + per);
        float qv[V], acc[V];
        T* fresh = reinterpret_cast<T*>(red + 4 * NW * 128);   // the new token's key and value of this head (behind the sums below)
        if (sp == S - 1) {
          if (tid < 2 * LPK) {   // ... and into the rings
            const int which = tid >= LPK, i = (tid - which * LPK) * V;
            uint4 v;
            take_vec(cur + ((1 + which) * d + i) * TB, tag, v);
            *reinterpret_cast<uint4*>((T*)(which ? L.v_ring : L.k_ring) + ((size_t)b * W + t % W) * d + h * hd + i) = v;
            *reinterpret_cast<uint4*>(fresh + which * hd + i) = v;
          }
          cons_bar();
        }
        uint4 q_raw;
        take_vec(cur + sub * V * TB, tag, q_raw);
        unpack(q_raw, qv, (T*)nullptr);
#pragma unroll
        for (int e = 0; e < V; e++) {
          qv[e] *= P.scale;
          acc[e] = 0.f;
        }
        const float slope = L.slopes[h];
        float mx = -INFINITY, den = 0.f;
        constexpr int U = 4;
#pragma unroll 1
        for (int base = k0 + warp * KPW; base < k1; base += NW * KPW * U) {
          uint4 kv[U], vv[U];
#pragma unroll
          for (int u = 0; u < U; u++) {
            const int kk = base + u * NW * KPW + grp, j = j_lo + kk;
            kv[u] = vv[u] = make_uint4(0, 0, 0, 0);
            if (kk < k1) {
              if (j == t) {   // the new token's key and value are still activations
                kv[u] = *reinterpret_cast<const uint4*>(fresh + sub * V);
                vv[u] = *reinterpret_cast<const uint4*>(fresh + hd + sub * V);
              } else {
                const size_t off = ((size_t)b * W + j % W) * d + h * hd + sub * V;
                kv[u] = ldnc16(kr + off);
                vv[u] = ldnc16(vr + off);
              }
            }
          }
          float sc[U];
#pragma unroll
          for (int u = 0; u < U; u++) {
            const int kk = base + u * NW * KPW + grp;
            float kf[V];
            unpack(kv[u], kf, (T*)nullptr);
            float dot = 0.f;
#pragma unroll
            for (int e = 0; e < V; e++) dot = fmaf(qv[e], kf[e], dot);
            for (int off = LPK / 2; off > 0; off >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, off);
            if (a.softcap > 0.f) {
              float th;   // bf16: hardware tanh, relative error 2^-11, below the rounding of the output
              if (sizeof(T) == 2) asm("tanh.approx.f32 %0, %1;" : "=f"(th) : "f"(dot * inv_cap));
              else th = tanhf(dot * inv_cap);
              dot = a.softcap * th;
            }
            sc[u] = kk < k1 ? dot - slope * (float)(nkeys - 1 - kk) : -INFINITY;
          }
          float mnew = mx;
#pragma unroll
          for (int u = 0; u < U; u++) mnew = fmaxf(mnew, sc[u]);
          if (mnew > -INFINITY) {
            const float corr = __expf(mx - mnew);
            den *= corr;
#pragma unroll
            for (int e = 0; e < V; e++) acc[e] *= corr;
#pragma unroll
            for (int u = 0; u < U; u++) {
              const float pw = __expf(sc[u] - mnew);
              float vf[V];
              unpack(vv[u], vf, (T*)nullptr);
              den += pw;
#pragma unroll
              for (int e = 0; e < V; e++) acc[e] = fmaf(pw, vf[e], acc[e]);
            }
            mx = mnew;
          }
        }
        // the groups of the CTA meet: [NG] maxima, [NG] denominators, [NG][hd] sums
        const int NG = NW * KPW, gi = warp * KPW + grp;
        float *gm = red, *gl = red + NG, *ga = red + 2 * NG;
        if (sub == 0) {
          gm[gi] = mx;
          gl[gi] = den;
        }
#pragma unroll
        for (int e = 0; e < V; e++) ga[gi * hd + sub * V + e] = acc[e];
        cons_bar();
        if (tid < hd) {
          float M = -INFINITY, num = 0.f, dn = 0.f;
          for (int i = 0; i < NG; i++) M = fmaxf(M, gm[i]);
#pragma unroll 4
          for (int i = 0; i < NG; i++) {
            const float mg = gm[i];
            const float w = mg > -INFINITY ? __expf(mg - M) : 0.f;
            num = fmaf(ga[i * hd + tid], w, num);
            dn = fmaf(gl[i], w, dn);
          }
          if (S == 1) {   // one range: the row of c_proj itself
            ((T*)att_at())[(size_t)b * d + h * hd + tid] = Elem<T>::from_f(num / dn);
          } else {
            float* out = att_at() + (size_t)it * (hd + 4);
            out[tid] = num;
            if (tid == 0) {
              out[hd] = M;
              out[hd + 1] = dn;
            }
          }
        }
        cons_bar();
      }
      if (cta < owners) arrive();
      continue;
    }

    // ================================================================ the rows of the product, in shared memory
    // (bf16: rows 64 bytes past a multiple of 128 apart: conflict-free fragments)
    const int K = sg.K;
    const int pitch = sizeof(T) == 2 ? ((min(K, xs_cols) * 2 + 127) & ~127) + 64 : min(K, xs_cols) * 4;
    const bool first = sg.layer == 0 && (kind == ST_STU || kind == ST_QKV);   // the rows are the step's input
    const bool arrives = kind == ST_GATE_UP ? !P.tagged_h : kind == ST_STU || kind == ST_CPROJ || kind == ST_DOWN ? !words_x : false;
    if (kind == ST_CPROJ && !wait(owners)) break;
    if (kind == ST_DOWN && !P.tagged_h && !wait(G)) break;
    if (normed && !first && !words_x && !wait(G)) break;
    if (r0 >= r1) {   // no feature of this product: its rows may be gone before they are looked at
      if (arrives) arrive();
      continue;
    }
    if (normed) {
      // The rows go to shared memory times the norm weight; the factor of a row's mean square, which is known when all of it has
      // been seen, goes onto its sums instead.
      const T* nw = (const T*)(kind == ST_LM_HEAD ? a.norm_final : kind == ST_GATE_UP ? L.norm2 : L.norm1);
      auto more = [&](int v) { return __ldg(reinterpret_cast<const uint2*>(nw) + v); };
      auto use = [&](float& ss, int m, int v, const uint2& val, const uint2& w) {
        float f[8 / sizeof(T)], g8[8 / sizeof(T)];
        unpack8(val, f, (T*)nullptr);
        unpack8(w, g8, (T*)nullptr);
#pragma unroll
        for (int j = 0; j < (int)(8 / sizeof(T)); j++) {
          ss += f[j] * f[j];
          f[j] *= g8[j];
        }
        *reinterpret_cast<uint2*>(xs + m * pitch + v * 8) = pack8(f, (T*)nullptr);
      };
      const char* words = rows_at(kind == ST_GATE_UP ? MID_ROWS : X_ROWS);
      const uint32_t tag_in = tag_of(kind == ST_GATE_UP ? sg.layer : sg.layer - 1);
      if constexpr (MM <= 2) {
        float ss[MM];
#pragma unroll
        for (int m = 0; m < MM; m++) ss[m] = 0.f;
        auto add = [&](int m, int v, const uint2& val, const uint2& w) {
#pragma unroll
          for (int mm = 0; mm < MM; mm++)
            if (mm == m) use(ss[mm], m, v, val, w);
        };
        if (first) {
#pragma unroll 1
          for (int v = tid; v < d * (int)sizeof(T) / 8; v += CONS) {
            const uint2 w = more(v);
#pragma unroll
            for (int m = 0; m < MM; m++)
              if (m < B) add(m, v, s_row[m] ? __ldcg(reinterpret_cast<const uint2*>(s_row[m]) + v) : make_uint2(0, 0), w);
          }
        } else {
          take(words, d, 0, d, 0, tag_in, more, add);
        }
        const float total = fold<MM>(ss, lane);   // of row lane / (32 / MM)
        if (lane % (32 / MM) == 0) s_part[lane / (32 / MM)][warp] = total;
      } else if (first || !words_x) {
        const T* rows = (const T*)words;
        float ss[MM];
#pragma unroll
        for (int m = 0; m < MM; m++) ss[m] = 0.f;
#pragma unroll 1
        for (int v = tid; v < d / V; v += CONS) {
          uint4 raw[MM];   // every row's piece is requested before the first is used
#pragma unroll
          for (int m = 0; m < MM; m++) {
            const T* row = m >= B ? nullptr : first ? s_row[m] : rows + (size_t)m * d;
            raw[m] = row ? ldcg16(row + v * V) : make_uint4(0, 0, 0, 0);
          }
          const uint2 w0 = more(2 * v), w1 = more(2 * v + 1);
#pragma unroll
          for (int m = 0; m < MM; m++)
            if (m < B) {
              use(ss[m], m, 2 * v, make_uint2(raw[m].x, raw[m].y), w0);
              use(ss[m], m, 2 * v + 1, make_uint2(raw[m].z, raw[m].w), w1);
            }
        }
        const float total = fold<MM>(ss, lane);   // of row lane / (32 / MM)
        if (lane % (32 / MM) == 0) s_part[lane / (32 / MM)][warp] = total;
      } else {
#pragma unroll 1
        for (int m0 = 0; m0 < (RG < MM ? B : 1); m0 += RG) {
          float ss[RG];
#pragma unroll
          for (int m = 0; m < RG; m++) ss[m] = 0.f;
          take(words, d, 0, d, m0, tag_in, more,
               [&](int m, int v, const uint2& val, const uint2& w) {
#pragma unroll
                 for (int mm = 0; mm < RG; mm++)
                   if (mm == m) use(ss[mm], m0 + m, v, val, w);
               });
          const float total = fold<RG>(ss, lane);   // of row m0 + lane / (32 / RG)
          if (lane % (32 / RG) == 0) s_part[m0 + lane / (32 / RG)][warp] = total;
        }
      }
    } else if (kind == ST_DOWN) {
      load_h(sg.layer, 0, min(K, xs_cols), pitch);
    } else if (S == 1) {
      load_plain((const T*)att_at(), K, 0, K, pitch);
    } else {   // ST_CPROJ: merge the key ranges of every head
      const int q4 = d / 4;
#pragma unroll 1
      for (int i = tid; i < B * q4; i += CONS) {
        const int m = i / q4, e = (i - m * q4) * 4, h = e / hd;
        const float* p = att_at() + (size_t)(m * H + h) * S * (hd + 4);
        float4 n4[8];
        float2 md[8];
#pragma unroll
        for (int s = 0; s < 8; s++)
          if (s < S) {
            n4[s] = __ldcg(reinterpret_cast<const float4*>(p + (size_t)s * (hd + 4) + (e - h * hd)));
            md[s] = __ldcg(reinterpret_cast<const float2*>(p + (size_t)s * (hd + 4) + hd));
          }
        float M = -INFINITY, dn = 0.f;
#pragma unroll
        for (int s = 0; s < 8; s++)
          if (s < S) M = fmaxf(M, md[s].x);
        float y[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int s = 0; s < 8; s++)
          if (s < S) {
            const float w = md[s].x > -INFINITY ? __expf(md[s].x - M) : 0.f;
            dn = fmaf(w, md[s].y, dn);
            y[0] = fmaf(n4[s].x, w, y[0]);
            y[1] = fmaf(n4[s].y, w, y[1]);
            y[2] = fmaf(n4[s].z, w, y[2]);
            y[3] = fmaf(n4[s].w, w, y[3]);
          }
        const float inv = 1.f / dn;
#pragma unroll
        for (int j = 0; j < 4; j++) y[j] *= inv;
        T* dst = reinterpret_cast<T*>(xs + m * pitch) + e;
#pragma unroll
        for (int j = 0; j < 4; j++) dst[j] = Elem<T>::from_f(y[j]);
      }
    }
    if (!go_on()) break;
    if (normed && tid < B) {   // (read behind the barrier at the end of the product)
      float s = 0.f;
#pragma unroll
      for (int w = 0; w < NW; w++) s += s_part[tid][w];
      s_scale[tid] = rsqrtf(s / (float)d + (kind == ST_LM_HEAD ? a.eps_final : kind == ST_GATE_UP ? L.eps2 : L.eps1));
    }

    // ================================================================ the product
    const uint32_t tag = tag_of(sg.layer);
    auto hand_on = [&](int rows, int m, int n, T v, uint32_t tag) {   // a value of the residual stream
      if (words_x) Tagged<T>::put(rows_at(rows + m), n, v, tag);
      else ((T*)rows_at(rows))[(size_t)m * d + n] = v;
    };
    auto finish = [&](int m, int n, float v, float v2) {   // m sequence, n feature; v2: the up projection
      if (normed) {
        v *= s_scale[m];
        v2 *= s_scale[m];
      }
      switch (kind) {
        case ST_STU: {
          const float xp = round_to<T>(v);
          ((T*)L.hist)[((size_t)((size_t)m * d + n) * 2 + par) * L.Lh + s_pos] = Elem<T>::from_f(xp);
          stream = round_to<T>(stream + round_to<T>(2.f * (s_hist[tid] + xp * tap0)));
          hand_on(MID_ROWS, m, n, Elem<T>::from_f(stream), tag);
          break;
        }
        case ST_QKV: Tagged<T>::put(rows_at(QKV_ROWS + 3 * m), n, Elem<T>::from_f(v), tag); break;
        case ST_CPROJ:
          stream = round_to<T>(stream + round_to<T>(v));
          hand_on(MID_ROWS, m, n, Elem<T>::from_f(stream), tag);
          break;
        case ST_GATE_UP: {
          const T h = Elem<T>::from_f(round_to<T>(gelu_tanh(round_to<T>(v))) * round_to<T>(v2));
          if (P.tagged_h) Tagged<T>::put(rows_at(H_ROWS) + (size_t)m * I * TB, n, h, tag);
          else ((T*)rows_at(H_ROWS))[(size_t)m * I + n] = h;
          break;
        }
        case ST_DOWN:
          stream = round_to<T>(stream + round_to<T>(v));
          hand_on(X_ROWS, m, n, Elem<T>::from_f(stream), tag);
          if (sg.layer == a.n_layers - 1) xbuf[(size_t)m * d + n] = Elem<T>::from_f(stream);
          break;
        default: ((T*)a.logits)[(size_t)m * a.ld_logits + n] = Elem<T>::from_f(v);
      }
    };
    const bool dual = kind == ST_GATE_UP;
    const int F = dual ? 8 : 16;
#pragma unroll 1
    for (int base = r0; base < r1; base += TILES * F) {   // tiles whose sums fit the buffer
      const int feats = min(TILES * F, r1 - base);
#pragma unroll 1
      for (int f = 0; f < feats; f += F) {
        const int nf = min(F, feats - f), rows = dual ? 2 * nf : nf;
        float* sums = red + (f / F) * (NW * 128);
        float acc[4][4];
#pragma unroll
        for (int c = 0; c < 4; c++) acc[0][c] = acc[1][c] = acc[2][c] = acc[3][c] = 0.f;
        const int pieces = sg.pieces == 1 ? 1 : rows == down_rows ? down_pieces : unit_pieces(rows, sg.pieces, slots, packed, xs_cols / d);
#pragma unroll 1
        for (int k0 = 0, p0 = 0; k0 < K; k0 += pieces * d, p0 += pieces, unit++) {
          const int np = min(pieces, sg.pieces - p0), n = rows * np, len = min(np * d, K - k0);
          if (slot + n > slots) slot = 0;
          const int kx = k0 < xs_cols ? k0 : k0 % xs_cols;   // column of the unit in the rows
          if (k0 && kx == 0) {   // the next columns of the rows (one tile only: own <= 32 features, see the host)
            cons_bar();
            load_h(sg.layer, k0, min(xs_cols, K - k0), pitch);
            cons_bar();
          }
          const unsigned char* rows0 = ring + (size_t)slot * pitch_w;
          const int row_pitch = np * pitch_w;
          tma::mbar_wait_bounded(&full_bar[unit % UNITS], (unit / UNITS) & 1u, &s_abort);
          if constexpr (sizeof(T) == 2) {
            // rows past the end of the unit: any row, their results are not used
            const unsigned char* lo_row = rows0 + (g < rows ? g * row_pitch : 0);
            const int rh = (dual ? nf : 8) + g;
            const unsigned char* hi_row = rows0 + (rh < rows ? rh * row_pitch : 0);
            const unsigned char* xrow = xs + g * pitch + kx * 2;
            const int nch = (len + 31) >> 5, last = len - 8 - q * 8;
            const unsigned char *lo_p = lo_row + q * 16, *hi_p = hi_row + q * 16, *x_p = xrow + q * 16;
#pragma unroll 1
            for (int c = warp; c < nch; c += 2 * NW) {
              uint4 lo[2], hi[2], xv[2];
#pragma unroll
              for (int u = 0; u < 2; u++) {
                lo[u] = hi[u] = xv[u] = make_uint4(0, 0, 0, 0);
                if ((c + u * NW) * 32 <= last) {   // (the end of a row may lie inside a chunk)
                  lo[u] = *reinterpret_cast<const uint4*>(lo_p + (c + u * NW) * 64);
                  hi[u] = *reinterpret_cast<const uint4*>(hi_p + (c + u * NW) * 64);
                  if (g < B) xv[u] = *reinterpret_cast<const uint4*>(x_p + (c + u * NW) * 64);
                }
              }
#pragma unroll
              for (int u = 0; u < 2; u++)
                if (c + u * NW < nch) {
                  mma_16816(acc[2 * u & 3], lo[u].x, hi[u].x, lo[u].y, hi[u].y, xv[u].x, xv[u].y);
                  mma_16816(acc[2 * u + 1 & 3], lo[u].z, hi[u].z, lo[u].w, hi[u].w, xv[u].z, xv[u].w);
                }
            }
          } else {
            // pairs of rows over teams of warps, the chunks of the unit over the wk warps of a team
            constexpr int NV = 2 * MM;
            const int wk = team_warps(rows), kw = warp % wk, teams = NW / wk;
#pragma unroll 1
            for (int r2 = (warp / wk) * 2; r2 < rows; r2 += teams * 2) {
              const unsigned char* wa = rows0 + r2 * row_pitch;
              const unsigned char* wb = rows0 + (r2 + 1 < rows ? r2 + 1 : r2) * row_pitch;
              const unsigned char* xr = xs + kx * 4;
              float v2[NV];
#pragma unroll
              for (int i = 0; i < NV; i++) v2[i] = 0.f;
#pragma unroll 2
              for (int k = (kw * 32 + lane) * 4; k + 4 <= len; k += wk * 128) {
                const float4 w0 = *reinterpret_cast<const float4*>(wa + k * 4);
                const float4 w1 = *reinterpret_cast<const float4*>(wb + k * 4);
#pragma unroll
                for (int m = 0; m < MM; m++)
                  if (m < B) {
                    const float4 xv = *reinterpret_cast<const float4*>(xr + m * pitch + k * 4);
                    v2[m] = fmaf(xv.x, w0.x, v2[m]);
                    v2[MM + m] = fmaf(xv.x, w1.x, v2[MM + m]);
                    v2[m] = fmaf(xv.y, w0.y, v2[m]);
                    v2[MM + m] = fmaf(xv.y, w1.y, v2[MM + m]);
                    v2[m] = fmaf(xv.z, w0.z, v2[m]);
                    v2[MM + m] = fmaf(xv.z, w1.z, v2[MM + m]);
                    v2[m] = fmaf(xv.w, w0.w, v2[m]);
                    v2[MM + m] = fmaf(xv.w, w1.w, v2[MM + m]);
                  }
              }
              const float v = fold<NV>(v2, lane);
              if (lane % (32 / NV) == 0) {   // the same lane adds up the pieces of a row
                float* at = sums + (kw * 16 + r2) * MM + lane / (32 / NV);
                *at = k0 ? *at + v : v;
              }
            }
          }
          __syncwarp();
          if (lane == 0) tma::mbar_arrive(&empty_bar[unit % UNITS]);
          slot += n;
        }
        if (sizeof(T) == 2)
#pragma unroll
          for (int c = 0; c < 4; c++) sums[warp * 128 + c * 32 + lane] = (acc[0][c] + acc[1][c]) + (acc[2][c] + acc[3][c]);
      }
      cons_bar();
#pragma unroll 1
      for (int e = tid; e < B * feats; e += CONS) {
        const int m = B == 1 ? 0 : e / feats, n = e - m * feats, i = dual ? n >> 3 : n >> 4, row = n & (F - 1);
        const float* sums = red + i * (NW * 128);
        float v = 0.f, v2 = 0.f;
        if (sizeof(T) == 2) {
          // row r, column m of a tile: lane (r % 8) * 4 + m / 2, register (r / 8) * 2 + m % 2
          const int at = ((row >> 3) * 2 + (m & 1)) * 32 + (row & 7) * 4 + (m >> 1);
#pragma unroll
          for (int w = 0; w < NW; w++) {
            v += sums[w * 128 + at];
            if (dual) v2 += sums[w * 128 + at + 64];   // row + 8
          }
        } else {
          const int nf = min(F, feats - i * F), wk = team_warps(dual ? 2 * nf : nf);
          for (int w = 0; w < wk; w++) {
            v += sums[(w * 16 + row) * MM + m];
            if (dual) v2 += sums[(w * 16 + nf + row) * MM + m];
          }
        }
        finish(m, base + n, v, v2);
      }
      if (base + feats < r1) cons_bar();   // the sums have been read
    }
    if (arrives) arrive();
  }
  __syncthreads();   // with the producer
  if (cta == 0 && !s_abort) {   // once every CTA has read the positions and the control words (long ago, but for idle ones)
    if (tid == 0) poll_count(started, G);
    if (go_on()) {
      for (int i = tid; i < a.n_layers * B; i += CONS) layers[i / B].pos[2 * (i % B)] = t + 1;
      if (tid == 0) {
        epoch_word[2] = P.signature;
        *epoch_word = epoch + 1;
      }
    }
  }
  if (tid == 0 && s_abort) {
    atomicExch(epoch_word + 1, 1);
    if (a.status) atomicExch(a.status, 12);
  }
}

template <typename T, int MM>
int launch_step(const Params& P, size_t smem, cudaStream_t st) {
  auto k = token_step_kernel<T, MM>;
  static SmemLimit limit;
  const cudaError_t granted = allow_smem((const void*)k, STEP_SMEM, limit);
  if (granted != cudaSuccess) return (int)granted;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(device_sm_count());
  cfg.blockDim = dim3(THREADS);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeCooperative;   // its CTAs wait for one another: all of them resident
  at[0].val.cooperative = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, k, P);
  if (e != cudaSuccess) return (int)e;
  STU_CHECK_LAUNCH();
  return STU_OK;
}

// Distances of the activation rows in shared memory and of the ring's row slots (see the kernel).
int row_pitch(int K, int dtype) { return dtype == STU_BF16 ? ((K * 2 + 127) & ~127) + 64 : K * 4; }
int slot_pitch(int d, int dtype) { return dtype == STU_BF16 && d >= 1536 ? row_pitch(d, dtype) : d * (dtype == STU_BF16 ? 2 : 4); }
// Columns of the activation rows held at a time: all, or (more than 56 KB of down-projection rows, one tile of features
// per CTA) as many pieces of d as fit 32 KB, so that the ring keeps its depth (8 rows of 6144 bf16 values would leave
// it 28 of 57 row slots: gate/up 13 us instead of 7).
int held_cols(int B, int d, int I, int dtype) {
  const int e = dtype == STU_BF16 ? 2 : 4, all = I > d ? I : d, sms = device_sm_count();
  if (I <= d || B * I * e <= 57344 || (d + sms - 1) / sms > 16) return all;
  int n = 32768 / (B * d * e);
  const int pieces = (I + d - 1) / d;
  if (n < 1) n = 1;
  return n >= pieces ? all : n * d;
}
int ring_slots(int B, int d, int I, int dtype) {
  const long long room = STEP_SMEM - RED_BYTES - (long long)B * row_pitch(held_cols(B, d, I, dtype), dtype) - 128;
  const long long n = room / slot_pitch(d, dtype);
  return n < 0 ? 0 : (n > 1024 ? 1024 : (int)n);
}

}  // namespace

// Bytes of the workspace of stu_token_step: 512 of control words (zero them once), the rows between the products and
// the attention items.
extern "C" long long stu_token_step_workspace_bytes(int d, int I, int H, int dtype) {
  if (d <= 0 || I <= 0 || H < 0) return 0;
  const long long e = dtype == STU_BF16 ? Tagged<bf16>::BYTES : Tagged<float>::BYTES, hd = H > 0 ? d / H : 0;
  return 512 + (40ll * d + 8ll * I) * e + (8ll * H + 160) * (hd + 4) * 4 + 256;
}

// 1 when stu_token_step takes a stack of these sizes, else 0.  H = 0: no attention layer.
extern "C" int stu_token_step_supported(int n_layers, int B, int d, int I, int H, int dtype) {
  if ((dtype != STU_BF16 && dtype != STU_F32) || n_layers < 1 || n_layers > MAXL) return 0;
  const int vec = dtype == STU_BF16 ? 8 : 4;
  if (B < 1 || B > 8 || d < 1 || I < 1 || d % vec || I % vec || H < 0) return 0;
  if (d > MAX_VECS * vec) return 0;
  if (H > 0) {
    if (d % H) return 0;
    const int lanes = d / H / vec;   // lanes per key
    if (d / H % vec || (lanes != 4 && lanes != 8 && lanes != 16 && lanes != 32) || d / H > CONS) return 0;
    if (B * H > 768) return 0;
  }
  const int sms = device_sm_count(), own = (d + sms - 1) / sms;
  if (own > MAX_ROWS || d > (1 << 22) || I > (1 << 22)) return 0;
  return ring_slots(B, d, I, dtype) >= 24 ? 1 : 0;
}

// Row slots of the weight ring that stu_token_step has for these sizes.
extern "C" int stu_token_step_ring_slots(int B, int d, int I, int dtype) {
  if ((dtype != STU_BF16 && dtype != STU_F32) || B < 1 || B > 8 || d < 1 || I < 1) return 0;
  return ring_slots(B, d, I, dtype);
}

extern "C" long long stu_token_step_plan_bytes(int n_layers) {
  return n_layers < 1 || n_layers > MAXL ? 0 : (5ll * n_layers + 1) * sizeof(Stage) + (long long)n_layers * sizeof(StuStepLayer);
}

// Checks the descriptors and writes the plan (stu_token_step_plan_bytes of host memory); the caller copies it to the
// device once.  Returns the number of stages, or an error (< 0).
extern "C" int stu_token_step_plan(const StuStepLayer* layers, const StuStepArgs* args, int dtype, void* plan) {
  if (!layers || !args || !plan) return STU_ERR_NULL;
  const StuStepArgs& a = *args;
  if (!stu_token_step_supported(a.n_layers, a.B, a.d, a.I, a.H, dtype)) return STU_ERR_UNSUPPORTED;
  if (a.lm_head && (!a.norm_final || a.V < 1)) return STU_ERR_NULL;
  if (a.V >= (1 << 24)) return STU_ERR_UNSUPPORTED;
  if (a.lm_head && (!aligned16(a.norm_final) || !aligned16(a.lm_head))) return STU_ERR_ALIGN;
  Stage* t = (Stage*)plan;
  for (int l = 0; l < a.n_layers; l++) {
    const StuStepLayer& L = layers[l];
    const bool attn = L.kind == STU_STEP_ATTENTION;
    if (L.kind != STU_STEP_STU && !attn) return STU_ERR_UNSUPPORTED;
    if (!L.norm1 || !L.w1 || !L.norm2 || !L.wg || !L.wu || !L.wd || !L.pos) return STU_ERR_NULL;
    if (attn ? (!L.wo || !L.k_ring || !L.v_ring || !L.slopes) : (!L.hist || !L.taps)) return STU_ERR_NULL;
    if (attn && (a.H < 1 || L.W < a.window + 1)) return STU_ERR_SHAPE;
    if (!attn && (L.Lh < 1 || L.Lh % 8)) return STU_ERR_SHAPE;
    const void* ptrs[] = {L.norm1, L.w1, L.norm2, L.wg, L.wu, L.wd, attn ? L.wo : L.hist, attn ? L.k_ring : L.taps,
                          attn ? L.v_ring : L.hist};
    for (const void* p : ptrs)
      if (!aligned16(p)) return STU_ERR_ALIGN;
    const short sl = (short)l;
    if (attn) {
      *t++ = {(const char*)L.w1, nullptr, 3 * a.d, a.d, ST_QKV, sl, 1};
      *t++ = {nullptr, nullptr, 0, 0, ST_ATTEND, sl, 1};
      *t++ = {(const char*)L.wo, nullptr, a.d, a.d, ST_CPROJ, sl, 1};
    } else {
      *t++ = {(const char*)L.w1, nullptr, a.d, a.d, ST_STU, sl, 1};
    }
    *t++ = {(const char*)L.wg, (const char*)L.wu, a.I, a.d, ST_GATE_UP, sl, 1};
    *t++ = {(const char*)L.wd, nullptr, a.d, a.I, ST_DOWN, sl, (a.I + a.d - 1) / a.d};
  }
  if (a.lm_head) *t++ = {(const char*)a.lm_head, nullptr, a.V, a.d, ST_LM_HEAD, (short)a.n_layers, 1};
  const int nst = (int)(t - (Stage*)plan);
  StuStepLayer* out = (StuStepLayer*)t;
  for (int l = 0; l < a.n_layers; l++) out[l] = layers[l];
  return nst;
}

// The producer's walk through the ring, on the host, for every CTA of the launch that stu_token_step would make of a plan
// (in host memory): 0, or 1 + the stage at whose unit a CTA would wait for slots that nothing is left to release.
extern "C" int stu_token_step_walk(const void* plan, int n_stages, const StuStepArgs* args, int dtype) {
  if (!plan || !args) return STU_ERR_NULL;
  const StuStepArgs& a = *args;
  if (!stu_token_step_supported(a.n_layers, a.B, a.d, a.I, a.H, dtype)) return STU_ERR_UNSUPPORTED;
  if (n_stages < 3 * a.n_layers || n_stages > 5 * a.n_layers + 1) return STU_ERR_SHAPE;
  const Stage* tab = (const Stage*)plan;
  const int slots = ring_slots(a.B, a.d, a.I, dtype), in_rows = held_cols(a.B, a.d, a.I, dtype) / a.d, sms = device_sm_count();
  const bool packed = slot_pitch(a.d, dtype) == a.d * (dtype == STU_BF16 ? 2 : 4);
  for (int cta = 0; cta < sms; cta++) {
    int slots_of[UNITS], head = 0, used = 0;
    unsigned issued = 0, freed = 0;
    for (int st = 0; st < n_stages; st++) {
      const Stage& s = tab[st];
      if (!s.W) continue;
      const bool dual = s.W2 != nullptr;
      const Range r = share_of(s.N, cta, sms);
      for (int f0 = r.r0, F = dual ? 8 : 16; f0 < r.r1; f0 += F) {
        const int nf = F < r.r1 - f0 ? F : r.r1 - f0, rows = dual ? 2 * nf : nf;
        const int pieces = s.pieces == 1 ? 1 : unit_pieces(rows, s.pieces, slots, packed, in_rows);
        for (int p0 = 0; p0 < s.pieces; p0 += pieces) {
          const int n = rows * (pieces < s.pieces - p0 ? pieces : s.pieces - p0);
          int skip = unit_skip(head, n, slots, used);
          while (used + skip + n > slots || issued - freed == UNITS) {
            if (freed == issued) return st + 1;
            used -= slots_of[freed++ % UNITS];
            skip = unit_skip(head, n, slots, used);
          }
          if (head + n > slots) head = 0;
          slots_of[issued++ % UNITS] = skip + n;
          head += n;
          used += skip + n;
        }
      }
    }
  }
  return 0;
}

extern "C" int stu_token_step(const void* plan, int n_stages, const StuStepArgs* args, int dtype, void* stream) {
  if (!plan || !args || !args->x || !args->workspace) return STU_ERR_NULL;
  const StuStepArgs& a = *args;
  if (!stu_token_step_supported(a.n_layers, a.B, a.d, a.I, a.H, dtype)) return STU_ERR_UNSUPPORTED;
  if (n_stages < 3 * a.n_layers || n_stages > 5 * a.n_layers + 1) return STU_ERR_SHAPE;
  if (a.workspace_bytes < stu_token_step_workspace_bytes(a.d, a.I, a.H, dtype)) return STU_ERR_SHAPE;
  if (((uintptr_t)a.workspace & 255u) || !aligned16(a.x) || !aligned16(plan)) return STU_ERR_ALIGN;
  if (a.ids && (!a.embedding || a.V < 1)) return STU_ERR_NULL;
  if (a.ids && !aligned16(a.embedding)) return STU_ERR_ALIGN;
  if (a.lm_head && !a.logits) return STU_ERR_NULL;
  Params P;
  P.a = a;
  P.plan = (const uint4*)plan;
  P.nst = n_stages;
  P.slots = ring_slots(a.B, a.d, a.I, dtype);
  P.xs_cols = held_cols(a.B, a.d, a.I, dtype);
  P.pitch = slot_pitch(a.d, dtype);
  P.scale = a.H > 0 ? 1.0f / sqrtf((float)(a.d / a.H)) : 1.f;
  P.tagged_x = (long long)a.B * a.d * (dtype == STU_BF16 ? Tagged<bf16>::BYTES : Tagged<float>::BYTES) <= TAGGED_X_BYTES;
  P.tagged_h = (long long)a.B * a.I * (dtype == STU_BF16 ? Tagged<bf16>::BYTES : Tagged<float>::BYTES) <= (a.B <= 2 ? TAGGED_H_BYTES : TAGGED_H_BYTES / 2);
  P.signature = (int)((((a.B * 64 + a.n_layers) * 1021 + a.H) * 65521u + (unsigned)a.d * 8191u + (unsigned)a.I) * 4u + (dtype == STU_BF16 ? 3u : 2u));
  const size_t smem = (((size_t)P.slots * P.pitch + 127) & ~(size_t)127) + RED_BYTES +
                      (size_t)a.B * row_pitch(P.xs_cols, dtype);
  cudaStream_t st = (cudaStream_t)stream;
  if (dtype == STU_BF16) {
    if (a.B == 1) return launch_step<bf16, 1>(P, smem, st);
    if (a.B == 2) return launch_step<bf16, 2>(P, smem, st);
    if (a.B <= 4) return launch_step<bf16, 4>(P, smem, st);
    return launch_step<bf16, 8>(P, smem, st);
  }
  if (a.B == 1) return launch_step<float, 1>(P, smem, st);
  if (a.B == 2) return launch_step<float, 2>(P, smem, st);
  if (a.B <= 4) return launch_step<float, 4>(P, smem, st);
  return launch_step<float, 8>(P, smem, st);
}
