// Flash-style attention on bf16 planes on the tensor cores (tcgen05), for head sizes up to 64 forward and of 64 backward: all heads of bf16
// operands, and those heads of Float32 operands that the half-precision planes of attention_half.cu would hold worse ("picked" ones).
//
// A Float32 value is cut into three bf16 planes by truncation (8 + 8 + 8 mantissa bits, any exponent: the split is exact); a bf16 operand is one
// plane.  The probabilities and dS have three.  A product is the sum of the plane products that lie above 2^-24 of it (six of three planes by
// three, three of three by one), the smallest ones first, accumulated in Float32 in tensor memory.  A bf16 tile in the 128-byte swizzle serves as K-major and as MN-major operand: a small kernel
// (`attn_split_kernel`; for picked heads the kernels that pick them) lays K, V, Q and dO out once per call as the images that the MMAs read from
// shared memory, and tiles arrive by plain bulk copies.  Head sizes below 64 are padded with zeros in those images; their zero 16-feature steps are skipped.
//
// (For bf16 operands two half-precision planes of the probabilities and dS, as attention_half.cu has them, take a third of these MMAs away, but hold
// 23 bits of a weight above 2^-29 and ever fewer below: forward 299 -> 274 us, dK / dV 471 -> 445, dQ 319 -> 330 for batch 8, 16 heads of 64,
// 2048 x 2048, causal.)  What bounds the kernels: an MMA with N = 64 takes 44 clocks where its multiplications need 32, and between
// the MMAs of a block the weights' arithmetic.
//
// A block is 64 keys (64 queries in the dK / dV kernel) against the 128 rows of a CTA; a thread of a compute warp owns
// one row (one TMEM lane).  Every mbarrier wait is bounded; when one runs out the kernel records 4002 (forward), 4003
// (dQ) or 4004 (dK / dV) in the context's device error word, all roles leave their loops, tensor memory is released and
// the kernel returns.
#include "attention_tc.cuh"

using namespace fb_atc;

namespace {

// 32 values of a thread's row into the three planes of an A operand: 16 columns each at t0, t1 and t2
__device__ __forceinline__ void store_planes32(uint32_t t0, uint32_t t1, uint32_t t2, const uint32_t* v) {
  uint32_t a[16], b[16], c[16];
#pragma unroll
  for (int e = 0; e < 16; ++e) split3(__uint_as_float(v[2 * e]), __uint_as_float(v[2 * e + 1]), a[e], b[e], c[e]);
  tc_st_32x32b_x16(t0, a);
  tc_st_32x32b_x16(t1, b);
  tc_st_32x32b_x16(t2, c);
}

// One row of a CTA's own operand into tensor memory: NP planes of 32 columns each (Float32 source: 3, bf16 source: 1).
// True when a value of it is not finite.
template <int NP>
__device__ __forceinline__ bool row_to_tmem(const void* src, int width, bool live, bool vec, uint32_t t_addr) {
  bool odd = false;
#pragma unroll
  for (int hf = 0; hf < 2; ++hf) {
    if (NP == 3) {
      uint32_t v[32];
      row_f32((const float*)src, 32 * hf, width, live, vec, v);
#pragma unroll
      for (int c = 0; c < 32; ++c) odd |= not_finite(v[c]);
      store_planes32(t_addr + 16u * hf, t_addr + 32u + 16u * hf, t_addr + 64u + 16u * hf, v);
    } else {
      uint32_t v[16];
#pragma unroll
      for (int c = 0; c < 16; c += 4) {   // bf16 head sizes are multiples of 8
        uint4 x = make_uint4(0u, 0u, 0u, 0u);
        if (live && 32 * hf + 2 * c < width) x = __ldg((const uint4*)((const uint16_t*)src + 32 * hf + 2 * c));
        v[c] = x.x; v[c + 1] = x.y; v[c + 2] = x.z; v[c + 3] = x.w;
      }
#pragma unroll
      for (int c = 0; c < 16; ++c) odd |= not_finite(v[c]) | not_finite(v[c] << 16);
      tc_st_32x32b_x16(t_addr + 16u * hf, v);
    }
  }
  return odd;
}

// The plane products of A (NA planes) and B (NB planes) from the smallest to the largest: 3 x 3 leaves out the three below
// 2^-24 of the whole.
template <int NA, int NB>
struct Prod {
  static constexpr int N = NA == 3 && NB == 3 ? 6 : NA == 3 ? 3 : 1;
  static __device__ __forceinline__ constexpr int a(int i) { return N == 6 ? (i == 0 ? 2 : i == 2 || i == 3 ? 1 : 0) : N == 3 ? 2 - i : 0; }
  static __device__ __forceinline__ constexpr int b(int i) { return N == 6 ? (i == 1 ? 2 : i == 2 || i == 4 ? 1 : 0) : 0; }
};

// instruction descriptors: D = F32, A = B = BF16, M = 128; B K-major (n columns = rows of the tile) or MN-major
__device__ __forceinline__ uint32_t idesc_bf16(int n, bool b_mn) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((b_mn ? 1u : 0u) << 16) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(QT >> 4) << 24);
}
// D = A B', A = NP planes in tensor memory (32 columns each), B = NP K-major planes; nks steps of 16 features
template <int NP>
__device__ __forceinline__ void mma_rows_t(uint32_t d, uint32_t a_tmem, uint32_t b_smem, int nks) {
  const uint64_t b0 = desc_k(b_smem);
  const uint32_t idesc = idesc_bf16(KT, false), hi = (uint32_t)(b0 >> 32);
  using P = Prod<NP, NP>;
#pragma unroll
  for (int i = 0; i < P::N; ++i)
#pragma unroll
    for (int ks = 0; ks < 4; ++ks)
      if (ks < nks)
        tc_mma_ta(d, a_tmem + (uint32_t)(32 * P::a(i) + 8 * ks), (uint32_t)b0 + (uint32_t)((P::b(i) * TILE + ks * 32) >> 4), hi, idesc,
                       (i > 0 || ks > 0) ? 1u : 0u);
}
// the same with A in shared memory: planes of 128 rows, 2 * TILE apart, all four steps (head sizes are zero-padded)
template <int NP>
__device__ __forceinline__ void mma_rows_s(uint32_t d, uint32_t a_smem, uint32_t b_smem) {
  const uint64_t a0 = desc_k(a_smem), b0 = desc_k(b_smem);
  const uint32_t idesc = idesc_bf16(KT, false), hi = (uint32_t)(a0 >> 32);
  using P = Prod<NP, NP>;
#pragma unroll
  for (int i = 0; i < P::N; ++i)
#pragma unroll
    for (int ks = 0; ks < 4; ++ks)
      tc_mma_sa(d, (uint32_t)a0 + (uint32_t)((P::a(i) * 2 * TILE + ks * 32) >> 4), (uint32_t)b0 + (uint32_t)((P::b(i) * TILE + ks * 32) >> 4),
                     hi, idesc, (i > 0 || ks > 0) ? 1u : 0u);
}
// D (+)= A B with A = three planes of 64 values in tensor memory that the compute warps stored in halves of 32 values:
// plane 0 at t01 + 32 half, plane 1 sixteen columns behind it, plane 2 at t2 + hstep2 half; B = NP MN-major planes whose K
// rows are the tile's rows; n columns (features, a multiple of 16)
template <int NP>
__device__ __forceinline__ void mma_planes(uint32_t d, uint32_t t01, uint32_t t2, uint32_t hstep2, uint32_t b_smem, int n, bool accumulate) {
  const uint64_t b0 = desc_mn(b_smem);
  const uint32_t idesc = idesc_bf16(n, true), hi = (uint32_t)(b0 >> 32);
  using P = Prod<3, NP>;
#pragma unroll
  for (int i = 0; i < P::N; ++i)
#pragma unroll
    for (int ks = 0; ks < 4; ++ks) {
      const uint32_t hf = (uint32_t)(ks >> 1), in = (uint32_t)(8 * (ks & 1));
      const uint32_t a = P::a(i) == 2 ? t2 + hstep2 * hf + in : t01 + 32u * hf + 16u * (uint32_t)P::a(i) + in;
      tc_mma_ta(d, a, (uint32_t)b0 + (uint32_t)((P::b(i) * TILE + ks * 2048) >> 4), hi, idesc, (accumulate || i > 0 || ks > 0) ? 1u : 0u);
    }
}

// -------------------------------------------------------------------------------------------- plane images ---
// One 64 x 64 tile of one (batch, head): bf16 rows -> the shared-memory image of the tile (row r at 128 r, its 16-byte chunks permuted by r & 7); rows past the end and features past the head size are 0.
// For dO the same pass forms what the softmax backward needs per query: {log2(e) lse, delta = sum_c dO_c O_c}; queries past
// the end get {inf, 0}, which makes their weights 0.
// Bound by memory.
struct SplitJob {
  const void* src;
  uint8_t* dst;
  int64_t L, E;
  int width, tiles;
};
struct SplitArgs {
  SplitJob job[4];
  const float* o;       // for the job of index 3 (dO)
  const float* lse;
  float2* rv;
  uint8_t* odd;         // [job][max_tiles] bytes, of odd_n per (batch, head): a value of the tile is not finite
  int H, vec, max_tiles, odd_n;
};

__global__ void __launch_bounds__(256) attn_split_kernel(SplitArgs A) {
  fb_after_previous();
  const SplitJob J = A.job[blockIdx.z];
  if ((int)blockIdx.x >= J.tiles) return;
  const int64_t bh = blockIdx.y;
  const int64_t b = bh / A.H;
  const int h = (int)(bh - b * A.H);
  uint8_t* dst = J.dst + (bh * J.tiles + blockIdx.x) * (int64_t)TILE;
  const int ch = threadIdx.x & 7;
  const bool is_do = blockIdx.z == 3;
  int odd = 0;
#pragma unroll
  for (int it = 0; it < 2; ++it) {
    const int r = (threadIdx.x >> 3) + 32 * it;
    const int64_t row = (int64_t)blockIdx.x * KT + r;
    const bool live = row < J.L;
    const int64_t off = (b * J.L + row) * J.E + (int64_t)h * J.width;
    uint8_t* out = dst + r * 128 + ((ch ^ (r & 7)) << 4);
    float x[8];
    uint4 t = make_uint4(0u, 0u, 0u, 0u);
    if (live && 8 * ch < J.width) t = __ldg((const uint4*)((const uint16_t*)J.src + off + 8 * ch));
    *(uint4*)out = t;
    const uint32_t w[4] = {t.x, t.y, t.z, t.w};
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      x[2 * e] = __uint_as_float(w[e] << 16);
      x[2 * e + 1] = __uint_as_float(w[e] & 0xffff0000u);
    }
#pragma unroll
    for (int e = 0; e < 8; ++e) odd |= not_finite(__float_as_uint(x[e])) ? 1 : 0;
    if (is_do) {
      float s = 0.0f;
#pragma unroll
      for (int e = 0; e < 8; e += 4) {
        if (!live || 8 * ch + e >= J.width) break;
        const float* po = A.o + off + 8 * ch + e;
        if (A.vec) {
          const float4 t = __ldg((const float4*)po);
          s = fmaf(x[e], t.x, s); s = fmaf(x[e + 1], t.y, s); s = fmaf(x[e + 2], t.z, s); s = fmaf(x[e + 3], t.w, s);
        } else {
          for (int u = 0; u < 4 && 8 * ch + e + u < J.width; ++u) s = fmaf(x[e + u], __ldg(po + u), s);
        }
      }
      s += __shfl_xor_sync(0xffffffffu, s, 1);
      s += __shfl_xor_sync(0xffffffffu, s, 2);
      s += __shfl_xor_sync(0xffffffffu, s, 4);
      if (ch == 0) A.rv[bh * ((int64_t)J.tiles * KT) + row] = live ? make_float2(A.lse[bh * J.L + row] * LOG2E, s) : make_float2(INFINITY, 0.0f);
    }
  }
  odd = __syncthreads_or(odd);
  if (threadIdx.x == 0) A.odd[bh * A.odd_n + (int)blockIdx.z * A.max_tiles + (int)blockIdx.x] = odd ? 1 : 0;
}

// --------------------------------------------------------------------------------------------- CTAs and items ---
struct Cta {
  uint8_t* smem;
  uint32_t sb, tmem;
  volatile uint32_t* s_tmem;
  volatile int* s_abort;
  int warp, lane;
};
// Kernels of picked heads have fewer CTAs than items (a tile of 128 rows of a head each), so that a launch that finds none is soon over: CTA c
// takes the items c, c + grid, ..., at most this many.  The heads of a tile follow one another, tiles with the most blocks under a causal mask
// first, so that CTAs with several items have about as much to do.  Each item has barriers of its own: arrivals of the one before may still
// be on their way.
constexpr int PICK_ITEMS = 8;
// a bit for each item of this CTA whose head is picked; the same in all warps
template <typename F>
__device__ __forceinline__ uint32_t picked_items(const uint8_t* pick, int64_t items, F head_of) {
  const int n = (int)(threadIdx.x & 31u);
  const int64_t item = blockIdx.x + (int64_t)n * gridDim.x;
  return __ballot_sync(0xffffffffu, n < PICK_ITEMS && item < items && pick[head_of(item)] != 0);
}
// Barriers (init, by one thread) and tensor memory; false, for all threads, after an earlier error.
template <typename F>
__device__ __forceinline__ bool cta_begin(Cta& c, uint8_t* smem_raw, uint32_t notes, uint32_t cols, const int32_t* dev_err, F init) {
  const Shared sh = aligned_smem(smem_raw);
  c.smem = sh.smem;
  c.sb = sh.sb;
  c.s_tmem = (volatile uint32_t*)(sh.smem + notes);
  c.s_abort = (volatile int*)(c.s_tmem + 1);
  volatile int* s_skip = (volatile int*)(c.s_tmem + 2);
  c.warp = uniform_warp();
  c.lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    init(sh.sb);
    *c.s_abort = 0;
    *s_skip = (*(volatile int32_t*)dev_err != 0) ? 1 : 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    fence_proxy_async();
  }
  __syncthreads();
  if (*s_skip != 0) return false;
  if (c.warp == 1) tmem_alloc(c.s_tmem, cols);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  c.tmem = __reduce_or_sync(0xffffffffu, *c.s_tmem);
  return true;
}
// Between two items: every load has been consumed and every product read.
__device__ __forceinline__ bool cta_next(const Cta& c) {
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  return *c.s_abort == 0;
}
__device__ __forceinline__ void cta_end(const Cta& c, uint32_t cols, int32_t* dev_err, int code) {
  tc_fence_before();
  __syncthreads();
  if (c.warp == 1) {
    __syncwarp();
    tmem_free(c.tmem, cols);
  }
  if (threadIdx.x == 0 && *c.s_abort != 0) atomicExch(dev_err, code);
}

// ------------------------------------------------------------------------------------------------------ forward ---
// One CTA owns 128 queries of one (batch, head); warp 0 copies K and V tiles into a ring of slots (K0 V0 K1 V1 ...),
// warp 1 issues the MMAs, warps 2-5 are the softmax (thread = query).  S = Q K' lands in 64 columns, the weights replace it
// as three planes (96 columns), P V lands in 64 more and is added to the thread's registers with round-to-nearest adds.
// Within a CTA these steps follow one another; what keeps the tensor pipe busy is the SECOND CTA on the SM: 256 of the 512
// TMEM columns, half of the registers and of shared memory each.
//   TMEM columns: Q planes 0..95, S -> P planes 96..191, P V 192..255
constexpr int FWD_THREADS = 192;
template <int NP>
struct FwdCfg {
  static constexpr int SLOTS = NP == 3 ? 4 : 8;
  enum { B_FULL = 0, B_FREE = SLOTS, B_QREADY = 2 * SLOTS, B_SFULL, B_PREADY, B_OFULL, B_COUNT };
  static constexpr int SLOT_BYTES = NP * TILE;
  static constexpr int BAR = SLOTS * SLOT_BYTES;
  static constexpr int NOTES = BAR + 8 * B_COUNT * (NP == 3 ? PICK_ITEMS : 1);
  static constexpr int SMEM = NOTES + 64 + 1024;
  static __device__ __forceinline__ void init(uint32_t bar0) {
    for (int s = 0; s < 2 * SLOTS; ++s) mbar_init(bar0 + 8u * (uint32_t)s, 1);
    mbar_init(bar0 + 8u * B_QREADY, 4);
    mbar_init(bar0 + 8u * B_SFULL, 1);
    mbar_init(bar0 + 8u * B_PREADY, 4);
    mbar_init(bar0 + 8u * B_OFULL, 1);
  }
};

// Queries i0 .. i0 + 127 of head h, batch entry b.
template <int NP>
__device__ __forceinline__ void fwd_item(const Cta& cta, uint32_t bar0, int64_t i0, int h, int64_t b, const void* __restrict__ qmat, const uint8_t* __restrict__ kimg,
                                         const uint8_t* __restrict__ vimg, float* __restrict__ o, uint16_t* __restrict__ o16, float* __restrict__ lse,
                                         uint8_t* __restrict__ odd_q, int odd_n, const AtcDims& D) {
  using cfg = FwdCfg<NP>;
  constexpr int S = cfg::SLOTS, B_FULL = cfg::B_FULL, B_FREE = cfg::B_FREE, B_QREADY = cfg::B_QREADY, B_SFULL = cfg::B_SFULL, B_PREADY = cfg::B_PREADY, B_OFULL = cfg::B_OFULL;
  const uint32_t sb = cta.sb, tmem = cta.tmem;
  volatile int* s_abort = cta.s_abort;
  const int warp = cta.warp, lane = cta.lane;
  auto bar = [&](int i) { return bar0 + 8u * (uint32_t)i; };
  const int64_t bh = b * D.H + h;
  int64_t kv_end = D.Lk;
  if (D.causal && i0 + QT < kv_end) kv_end = i0 + QT;
  const int nkb = (int)((kv_end + KT - 1) / KT);
  constexpr uint32_t T_R = 96, T_O = 192;

  if (warp == 0) {
    // ---------------------------------------------------------------- producer ---
    if (lane == 0) {
      const int64_t base = bh * D.ktiles * (int64_t)cfg::SLOT_BYTES;
      for (int n = 0; n < 2 * nkb; ++n) {
        const int s = n % S;
        if (n >= S && !mbar_wait(bar(B_FREE + s), (uint32_t)(n / S - 1) & 1u, s_abort)) break;
        mbar_arrive_expect_tx(bar(B_FULL + s), (uint32_t)cfg::SLOT_BYTES);
        bulk_load(sb + (uint32_t)(s * cfg::SLOT_BYTES), ((n & 1) ? vimg : kimg) + base + (int64_t)(n >> 1) * cfg::SLOT_BYTES,
                  (uint32_t)cfg::SLOT_BYTES, bar(B_FULL + s));
      }
    }
  } else if (warp == 1) {
    // -------------------------------------------------------------- MMA issuer ---
    {
      const int nks = (D.d + 15) >> 4, nv = (D.dv + 15) & ~15;
      auto issue_s = [&](int j) -> bool {
        const int n = 2 * j, s = n % S;
        if (!warp_wait(bar(B_FULL + s), (uint32_t)(n / S) & 1u, s_abort)) return false;
        tc_fence_after();
        mma_rows_t<NP>(tmem + T_R, tmem, sb + (uint32_t)(s * cfg::SLOT_BYTES), nks);
        tc_commit(bar(B_SFULL));
        tc_commit(bar(B_FREE + s));
        return true;
      };
      bool ok = warp_wait(bar(B_QREADY), 0u, s_abort) && issue_s(0);
      for (int j = 0; j < nkb && ok; ++j) {
        const int n = 2 * j + 1, s = n % S;
        ok = warp_wait(bar(B_FULL + s), (uint32_t)(n / S) & 1u, s_abort) && warp_wait(bar(B_PREADY), (uint32_t)j & 1u, s_abort);
        if (!ok) break;
        tc_fence_after();
        mma_planes<NP>(tmem + T_O, tmem + T_R, tmem + T_R + 64u, 16u, sb + (uint32_t)(s * cfg::SLOT_BYTES), nv, false);
        tc_commit(bar(B_OFULL));
        tc_commit(bar(B_FREE + s));
        // the next scores go where the weights are: the tensor pipe runs in order
        if (j + 1 < nkb) ok = issue_s(j + 1);
      }
    }
  } else {
    // ------------------------------------------------------------ softmax warps ---
    const int q = warp & 3;
    const int64_t gi = i0 + 32 * q + lane;
    const bool live = gi < D.Lq;
    const uint32_t t_row = tmem + ((uint32_t)(32 * q) << 16);
    const int64_t el = NP == 3 ? 4 : 2;
    const bool odd = row_to_tmem<NP>((const uint8_t*)qmat + el * ((b * D.Lq + gi) * D.E + (int64_t)h * D.d), D.d, live, D.vec != 0, t_row);
    const bool any = __any_sync(0xffffffffu, odd);
    if (NP == 1 && lane == 0) odd_q[bh * odd_n + (int)(i0 / QT) * 4 + q] = any ? 1 : 0;
    tc_wait_st();
    tc_fence_before();
    __syncwarp();
    if (lane == 0) mbar_arrive(bar(B_QREADY));
    float m = -INFINITY, l = 0.0f;
    float acc[HD];
#pragma unroll
    for (int c = 0; c < HD; ++c) acc[c] = 0.0f;
    // adds P V of block j to the accumulators (waits for its MMAs)
    auto add_pv = [&](int j) -> bool {
      if (!mbar_wait(bar(B_OFULL), (uint32_t)j & 1u, s_abort)) return false;
      tc_fence_after();
#pragma unroll
      for (int hf = 0; hf < 2; ++hf) {
        uint32_t v[32];
        tc_ld_32x32b_x32(t_row + T_O + 32u * hf, v);
        tc_wait_ld();
#pragma unroll
        for (int c = 0; c < 32; ++c) acc[32 * hf + c] += __uint_as_float(v[c]);
      }
      return true;
    };
    bool ok = true;
    for (int j = 0; j < nkb && ok; ++j) {
      // P V of the block before joins the accumulators while the tensor cores compute these scores
      ok = (j == 0 || add_pv(j - 1)) && mbar_wait(bar(B_SFULL), (uint32_t)j & 1u, s_abort);
      if (!ok) break;
      tc_fence_after();
      const int64_t j0 = (int64_t)j * KT;
      uint32_t s0[32], s1[32];
      tc_ld_32x32b_x32(t_row + T_R, s0);
      tc_ld_32x32b_x32(t_row + T_R + 32u, s1);
      tc_wait_ld();
      int64_t lim = D.Lk - j0;
      if (D.causal && gi - j0 + 1 < lim) lim = gi - j0 + 1;
      const int nvalid = lim < 0 ? 0 : (lim > KT ? KT : (int)lim);
      // keys the query may not see get a score of -inf (whole blocks below the diagonal need no test)
      if (nvalid < KT) {
#pragma unroll
        for (int c = 0; c < 32; ++c) {
          if (c >= nvalid) s0[c] = 0xff800000u;
          if (c + 32 >= nvalid) s1[c] = 0xff800000u;
        }
      }
      float mx0 = -INFINITY, mx1 = -INFINITY;
#pragma unroll
      for (int c = 0; c < 32; ++c) {
        mx0 = fmaxf(mx0, __uint_as_float(s0[c]));
        mx1 = fmaxf(mx1, __uint_as_float(s1[c]));
      }
      const float m_new = fmaxf(m, fmaxf(mx0, mx1));
      const float m_use = (m_new == -INFINITY) ? 0.0f : m_new;
      const float alpha = fast_exp2((m - m_use) * D.scale_log2);   // m = -inf gives 0
      const float mc = m_use * D.scale_log2;
      float rs0 = 0.0f, rs1 = 0.0f;
#pragma unroll
      for (int c = 0; c < 32; ++c) {
        const float p = fast_exp2(fmaf(__uint_as_float(s0[c]), D.scale_log2, -mc));
        rs0 += p;
        s0[c] = __float_as_uint(p);
      }
      store_planes32(t_row + T_R, t_row + T_R + 16u, t_row + T_R + 64u, s0);
#pragma unroll
      for (int c = 0; c < 32; ++c) {
        const float p = fast_exp2(fmaf(__uint_as_float(s1[c]), D.scale_log2, -mc));
        rs1 += p;
        s1[c] = __float_as_uint(p);
      }
      store_planes32(t_row + T_R + 32u, t_row + T_R + 48u, t_row + T_R + 80u, s1);
      tc_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar(B_PREADY));
      l = l * alpha + (rs0 + rs1);
      m = m_new;
      if (alpha != 1.0f) {   // the running maximum moved (rare after the first blocks)
#pragma unroll
        for (int c = 0; c < HD; ++c) acc[c] *= alpha;
      }
    }
    if (ok) ok = add_pv(nkb - 1);
    if (ok && live) {
      const float inv = l > 0.0f ? 1.0f / l : 0.0f;
      const int64_t off = (b * D.Lq + gi) * D.Ev + (int64_t)h * D.dv;
#pragma unroll
      for (int hf = 0; hf < 2; ++hf) {
        if (NP == 3 || o != nullptr) store_row32<false>(o + off, 32 * hf, D.dv, D.vec != 0, acc + 32 * hf, inv);
        if (NP == 1) store_row32<true>(o16 + off, 32 * hf, D.dv, true, acc + 32 * hf, inv);
      }
      lse[bh * D.Lq + gi] = (l > 0.0f) ? m * D.scale + logf(l) : -INFINITY;
    }
  }
}

__global__ void __launch_bounds__(FWD_THREADS, 2)
attn_fwd_tc_kernel(const uint16_t* __restrict__ q, const uint8_t* __restrict__ kimg, const uint8_t* __restrict__ vimg, float* __restrict__ o,
                   uint16_t* __restrict__ o16, float* __restrict__ lse, uint8_t* __restrict__ odd_q, int odd_n, AtcDims D, int32_t* __restrict__ dev_err) {
  fb_after_previous();
  extern __shared__ uint8_t smem_raw[];
  Cta cta;
  if (!cta_begin(cta, smem_raw, FwdCfg<1>::NOTES, 256u, dev_err, [](uint32_t sb) { FwdCfg<1>::init(sb + FwdCfg<1>::BAR); })) return;
  // causal: the last query tiles have the most key blocks, so they are scheduled first
  const int64_t i0 = (int64_t)(D.causal ? gridDim.x - 1 - blockIdx.x : blockIdx.x) * QT;
  fwd_item<1>(cta, cta.sb + FwdCfg<1>::BAR, i0, (int)blockIdx.y, (int64_t)blockIdx.z, q, kimg, vimg, o, o16, lse, odd_q, odd_n, D);
  cta_end(cta, 256u, dev_err, 4002);
}

// Float32 heads, picked ones
__global__ void __launch_bounds__(FWD_THREADS, 2)
attn_fwd_picked_kernel(const float* __restrict__ q, const uint8_t* __restrict__ kimg, const uint8_t* __restrict__ vimg, float* __restrict__ o, float* __restrict__ lse,
                       const uint8_t* __restrict__ pick, int64_t items, AtcDims D, int32_t* __restrict__ dev_err) {
  fb_after_previous();
  fb_let_next_start();
  extern __shared__ uint8_t smem_raw[];
  const int tiles = D.qtiles / 2;
  const int64_t heads = items / tiles;
  auto head_of = [&](int64_t item) { return item % heads; };
  const uint32_t mine = picked_items(pick, items, head_of);
  if (mine == 0) return;
  using cfg = FwdCfg<3>;
  auto bars = [](uint32_t sb, int n) { return sb + (uint32_t)(cfg::BAR + 8 * cfg::B_COUNT * n); };
  Cta cta;
  if (!cta_begin(cta, smem_raw, cfg::NOTES, 256u, dev_err, [&](uint32_t sb) {
        for (int n = 0; n < PICK_ITEMS; ++n) cfg::init(bars(sb, n));
      }))
    return;
  for (int n = 0; n < PICK_ITEMS; ++n) {
    if (!(mine >> n & 1)) continue;
    const int64_t item = blockIdx.x + (int64_t)n * gridDim.x, bh = head_of(item), b = bh / D.H;
    fwd_item<3>(cta, bars(cta.sb, n), (tiles - 1 - item / heads) * QT, (int)(bh - b * D.H), b, q, kimg, vimg, o, nullptr, lse, nullptr, 0, D);
    if (!cta_next(cta)) break;
  }
  cta_end(cta, 256u, dev_err, 4002);
}

// ----------------------------------------------------------------------------------------------------------- dQ ---
// One CTA owns 128 queries of one (batch, head).  Q and dO of those queries live in tensor memory for the whole kernel.
// For every block of 64 keys: S = Q K' and dP = dO V', the compute warps turn them into dS = P (dP - delta) with
// P = exp(S / sqrt(d) - lse) and put its planes over them, and dQ += dS K with the same K tile read MN-major.  Two S / dP
// regions and two sets of four compute warps take the blocks in turn: the tensor cores work on block j + 1 and on dQ of
// block j - 1 while a set is busy with block j.  dQ accumulates in tensor memory over at most 32 blocks (2048 keys: the
// adds truncate).
//   TMEM columns: Q planes 0..95, dO planes 96..191, two regions of 128 (S, dP -> dS planes) 192..447, dQ 448..511
template <int NP>
struct DqCfg {
  static constexpr int SLOTS = NP == 3 ? 4 : 6;
  enum { B_FULL = 0, B_FREE = SLOTS, B_QREADY = 2 * SLOTS, B_SFULL, B_DSREADY = B_SFULL + 2, B_DONE = B_DSREADY + 2, B_COUNT };
  static constexpr int SLOT_BYTES = 2 * NP * TILE;   // K tile, V tile
  static constexpr int BAR = SLOTS * SLOT_BYTES;
  static constexpr int NOTES = BAR + 8 * B_COUNT * (NP == 3 ? PICK_ITEMS : 1);
  static constexpr int SMEM = NOTES + 64 + 1024;
  static __device__ __forceinline__ void init(uint32_t bar0) {
    for (int s = 0; s < B_COUNT; ++s) mbar_init(bar0 + 8u * (uint32_t)s, s == B_QREADY ? 8 : s == B_DSREADY || s == B_DSREADY + 1 ? 4 : 1);
  }
};

template <int NP>
__device__ __forceinline__ void dq_item(const Cta& cta, uint32_t bar0, int64_t i0, int h, int64_t b, const void* __restrict__ q, const void* __restrict__ dout,
                                        const uint8_t* __restrict__ kimg, const uint8_t* __restrict__ vimg, const float2* __restrict__ rv, void* __restrict__ dq,
                                        const AtcDims& D) {
  using cfg = DqCfg<NP>;
  constexpr int S = cfg::SLOTS, B_FULL = cfg::B_FULL, B_FREE = cfg::B_FREE, B_QREADY = cfg::B_QREADY, B_SFULL = cfg::B_SFULL, B_DSREADY = cfg::B_DSREADY, B_DONE = cfg::B_DONE;
  const uint32_t sb = cta.sb, tmem = cta.tmem;
  volatile int* s_abort = cta.s_abort;
  const int warp = cta.warp, lane = cta.lane;
  auto bar = [&](int i) { return bar0 + 8u * (uint32_t)i; };
  const int64_t bh = b * D.H + h;
  int64_t kv_end = D.Lk;
  if (D.causal && i0 + QT < kv_end) kv_end = i0 + QT;
  const int nkb = (int)((kv_end + KT - 1) / KT);
  constexpr uint32_t T_DO = 96, T_R = 192, T_DQ = 448;

  if (warp == 0) {
    // ---------------------------------------------------------------- producer ---
    if (lane == 0) {
      const int64_t base = bh * D.ktiles * (int64_t)(NP * TILE);
      for (int j = 0; j < nkb; ++j) {
        const int s = j % S;
        if (j >= S && !mbar_wait(bar(B_FREE + s), (uint32_t)(j / S - 1) & 1u, s_abort)) break;
        mbar_arrive_expect_tx(bar(B_FULL + s), (uint32_t)cfg::SLOT_BYTES);
        const uint32_t dst = sb + (uint32_t)(s * cfg::SLOT_BYTES);
        const int64_t off = base + (int64_t)j * (NP * TILE);
        bulk_load(dst, kimg + off, NP * TILE, bar(B_FULL + s));
        bulk_load(dst + NP * TILE, vimg + off, NP * TILE, bar(B_FULL + s));
      }
    }
  } else if (warp == 1) {
    // -------------------------------------------------------------- MMA issuer ---
    {
      const int nks = (D.d + 15) >> 4, nvs = (D.dv + 15) >> 4, nd = (D.d + 15) & ~15;
      bool ok = warp_wait(bar(B_QREADY), 0u, s_abort);
      // step j: S and dP of block j + 2 (j >= -2) behind dQ of block j, whose planes they overwrite: the tensor pipe runs
      // in order
      for (int j = -2; j < nkb && ok; ++j) {
        if (j >= 0) {
          ok = warp_wait(bar(B_DSREADY + (j & 1)), (uint32_t)(j >> 1) & 1u, s_abort);
          if (!ok) break;
          tc_fence_after();
          const uint32_t r = tmem + T_R + (uint32_t)(128 * (j & 1));
          mma_planes<NP>(tmem + T_DQ, r, r + 64u, 32u, sb + (uint32_t)((j % S) * cfg::SLOT_BYTES), nd, j > 0);
          tc_commit(bar(B_FREE + j % S));
          if (j == nkb - 1) tc_commit(bar(B_DONE));
        }
        const int t = j + 2, s = t % S;
        if (t < nkb) {
          ok = warp_wait(bar(B_FULL + s), (uint32_t)(t / S) & 1u, s_abort);
          if (!ok) break;
          tc_fence_after();
          const uint32_t base = sb + (uint32_t)(s * cfg::SLOT_BYTES), r = tmem + T_R + (uint32_t)(128 * (t & 1));
          mma_rows_t<NP>(r, tmem, base, nks);
          mma_rows_t<NP>(r + 64u, tmem + T_DO, base + NP * TILE, nvs);
          tc_commit(bar(B_SFULL + (t & 1)));
        }
      }
    }
  } else {
    // ------------------------------------------------------------ compute warps ---
    const int set = (warp - 2) >> 2, qd = warp & 3;
    const int64_t gi = i0 + 32 * qd + lane;
    const bool live = gi < D.Lq;
    const uint32_t t_row = tmem + ((uint32_t)(32 * qd) << 16);
    const int64_t el = NP == 3 ? 4 : 2;
    // the first set brings Q into tensor memory, the second dO
    if (set == 0) row_to_tmem<NP>((const uint8_t*)q + el * ((b * D.Lq + gi) * D.E + (int64_t)h * D.d), D.d, live, D.vec != 0, t_row);
    else row_to_tmem<NP>((const uint8_t*)dout + el * ((b * D.Lq + gi) * D.Ev + (int64_t)h * D.dv), D.dv, live, D.vec != 0, t_row + T_DO);
    tc_wait_st();
    tc_fence_before();
    __syncwarp();
    if (lane == 0) mbar_arrive(bar(B_QREADY));
    const float2 ld = rv[bh * ((int64_t)D.qtiles * KT) + gi];   // {inf, 0} past the end: the weights become 0
    bool ok = true;
    for (int j = set; j < nkb && ok; j += 2) {
      ok = mbar_wait(bar(B_SFULL + set), (uint32_t)(j >> 1) & 1u, s_abort);
      if (!ok) break;
      tc_fence_after();
      const int64_t j0 = (int64_t)j * KT;
      int64_t lim = D.Lk - j0;
      if (D.causal && gi - j0 + 1 < lim) lim = gi - j0 + 1;
      const int nvalid = lim < 0 ? 0 : (lim > KT ? KT : (int)lim);
      const uint32_t r = t_row + T_R + (uint32_t)(128 * set);
#pragma unroll
      for (int hf = 0; hf < 2; ++hf) {
        uint32_t sv[32], dp[32];
        tc_ld_32x32b_x32(r + 32u * hf, sv);
        tc_ld_32x32b_x32(r + 64u + 32u * hf, dp);
        tc_wait_ld();
        if (nvalid >= KT) {
#pragma unroll
          for (int c = 0; c < 32; ++c)
            sv[c] = __float_as_uint(fast_exp2(fmaf(__uint_as_float(sv[c]), D.scale_log2, -ld.x)) * (__uint_as_float(dp[c]) - ld.y));
        } else {
#pragma unroll
          for (int c = 0; c < 32; ++c) {
            float p = fast_exp2(fmaf(__uint_as_float(sv[c]), D.scale_log2, -ld.x));
            if (c + 32 * hf >= nvalid) p = 0.0f;
            sv[c] = __float_as_uint(p * (__uint_as_float(dp[c]) - ld.y));
          }
        }
        // columns this thread has read already: 32 hf .. and 64 + 32 hf ..
        store_planes32(r + 32u * hf, r + 32u * hf + 16u, r + 64u + 32u * hf, sv);
      }
      tc_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar(B_DSREADY + set));
    }
    // each set writes 32 columns
    if (ok) ok = mbar_wait(bar(B_DONE), 0u, s_abort);
    if (ok) {
      tc_fence_after();
      uint32_t v[32];
      tc_ld_32x32b_x32(t_row + T_DQ + 32u * set, v);
      tc_wait_ld();
      if (live)
        store_row32<NP == 1>((uint8_t*)dq + el * ((b * D.Lq + gi) * D.E + (int64_t)h * D.d), 32 * set, D.d, D.vec != 0, (const float*)v, D.scale);
    }
  }
}

__global__ void __launch_bounds__(BWD_THREADS, 1)
attn_bwd_dq_tc_kernel(const uint16_t* __restrict__ q, const uint16_t* __restrict__ dout, const uint8_t* __restrict__ kimg, const uint8_t* __restrict__ vimg,
                      const float2* __restrict__ rv, uint16_t* __restrict__ dq, AtcDims D, int32_t* __restrict__ dev_err) {
  fb_after_previous();
  extern __shared__ uint8_t smem_raw[];
  Cta cta;
  if (!cta_begin(cta, smem_raw, DqCfg<1>::NOTES, 512u, dev_err, [](uint32_t sb) { DqCfg<1>::init(sb + DqCfg<1>::BAR); })) return;
  const int64_t i0 = (int64_t)(D.causal ? gridDim.x - 1 - blockIdx.x : blockIdx.x) * QT;
  dq_item<1>(cta, cta.sb + DqCfg<1>::BAR, i0, (int)blockIdx.y, (int64_t)blockIdx.z, q, dout, kimg, vimg, rv, dq, D);
  cta_end(cta, 512u, dev_err, 4003);
}

// ------------------------------------------------------------------------------------------------------ dK, dV ---
// Transposed, so that keys are the rows (TMEM lanes) of every accumulator.  One CTA owns 128 keys of one (batch, head); K
// and V stay in shared memory as A operands.  For every block of 64 queries:
//   S' = K Q'  and  dP' = V dO'    (B operands: the Q and dO tiles, K-major)
//   P' = exp(S' / sqrt(d) - lse_q),  dS' = P' (dP' - delta_q)     (compute warps; planes back into tensor memory)
//   dV += P' dO  and  dK += dS' Q   (B operands: the same Q and dO tiles, MN-major)
// As in the dQ kernel two regions and two sets of compute warps take the blocks in turn.  The ring of five tile slots
// holds dO0 Q0 dO1 Q1 dO2 ...; dV is issued before dK and dP' before S', so that a slot freed by dV of block i is
// reloaded (with Q of block i + 2) under dK of block i and dP' of block i + 2.  K and V in tensor memory would leave room
// for one region only; from shared memory an MMA of 128 x 64 x 16 takes 48 clocks, from tensor memory 44.
//   TMEM columns: two regions of 192 (S', dP', 64 more -> P' and dS' planes) 0..383, dV 384..447, dK 448..511
template <int NP>
struct KvCfg {
  static constexpr int SLOTS = NP == 3 ? 5 : 8;
  enum { B_FULL = 0, B_FREE = SLOTS, B_KV = 2 * SLOTS, B_SFULL, B_PREADY = B_SFULL + 2, B_DONE = B_PREADY + 2, B_COUNT };
  static constexpr int SLOT_BYTES = NP * TILE + 1024;   // a tile and, behind dO, {lse, delta} of its 64 queries
  static constexpr int K_OFF = SLOTS * SLOT_BYTES, V_OFF = K_OFF + NP * 2 * TILE;
  static constexpr int BAR = V_OFF + NP * 2 * TILE;
  static constexpr int NOTES = BAR + 8 * B_COUNT * (NP == 3 ? PICK_ITEMS : 1);
  static constexpr int SMEM = NOTES + 64 + 1024;
  static __device__ __forceinline__ void init(uint32_t bar0) {
    for (int s = 0; s < B_COUNT; ++s) mbar_init(bar0 + 8u * (uint32_t)s, s == B_PREADY || s == B_PREADY + 1 ? 4 : 1);
  }
};

// Keys j0 .. j0 + 127 of head h, batch entry b.
template <int NP>
__device__ __forceinline__ void dkdv_item(const Cta& cta, uint32_t bar0, int64_t j0, int h, int64_t b, const uint8_t* __restrict__ qimg, const uint8_t* __restrict__ doimg,
                                          const uint8_t* __restrict__ kimg, const uint8_t* __restrict__ vimg, const float2* __restrict__ rv, void* __restrict__ dk,
                                          void* __restrict__ dv, const AtcDims& D) {
  using cfg = KvCfg<NP>;
  constexpr int S = cfg::SLOTS, B_FULL = cfg::B_FULL, B_FREE = cfg::B_FREE, B_KV = cfg::B_KV, B_SFULL = cfg::B_SFULL, B_PREADY = cfg::B_PREADY, B_DONE = cfg::B_DONE;
  const uint32_t sb = cta.sb, tmem = cta.tmem;
  volatile int* s_abort = cta.s_abort;
  const int warp = cta.warp, lane = cta.lane;
  auto bar = [&](int i) { return bar0 + 8u * (uint32_t)i; };
  const int64_t bh = b * D.H + h;
  // query blocks that see these keys: all of them, or under a causal mask those from the diagonal on
  const int ib0 = D.causal ? (int)(j0 / KT) : 0;
  const int nqb = (int)((D.Lq + KT - 1) / KT) - ib0;   // may be <= 0: nothing attends to these keys
  constexpr uint32_t T_DV = 384, T_DK = 448;

  if (warp == 0) {
    // ---------------------------------------------------------------- producer ---
    if (lane == 0 && nqb > 0) {
      mbar_arrive_expect_tx(bar(B_KV), (uint32_t)(4 * NP * TILE));
#pragma unroll
      for (int p = 0; p < NP; ++p)
#pragma unroll
        for (int t = 0; t < 2; ++t) {   // plane p of the CTA's two 64-key tiles, one after the other
          const int64_t off = ((bh * D.ktiles + j0 / KT + t) * NP + p) * (int64_t)TILE;
          bulk_load(sb + (uint32_t)(cfg::K_OFF + (2 * p + t) * TILE), kimg + off, TILE, bar(B_KV));
          bulk_load(sb + (uint32_t)(cfg::V_OFF + (2 * p + t) * TILE), vimg + off, TILE, bar(B_KV));
        }
      for (int n = 0; n < 2 * nqb; ++n) {
        const int s = n % S;
        if (n >= S && !mbar_wait(bar(B_FREE + s), (uint32_t)(n / S - 1) & 1u, s_abort)) break;
        const bool is_do = (n & 1) == 0;
        const int64_t tile = bh * D.qtiles + ib0 + (n >> 1);
        const uint32_t dst = sb + (uint32_t)(s * cfg::SLOT_BYTES);
        mbar_arrive_expect_tx(bar(B_FULL + s), (uint32_t)(NP * TILE + (is_do ? 512 : 0)));
        bulk_load(dst, (is_do ? doimg : qimg) + tile * (int64_t)(NP * TILE), NP * TILE, bar(B_FULL + s));
        if (is_do) bulk_load(dst + NP * TILE, rv + tile * KT, 512u, bar(B_FULL + s));
      }
    }
  } else if (warp == 1) {
    // -------------------------------------------------------------- MMA issuer ---
    if (nqb > 0) {
      const int nd = (D.d + 15) & ~15, nv = (D.dv + 15) & ~15;
      auto slot = [&](int n) { return sb + (uint32_t)((n % S) * cfg::SLOT_BYTES); };
      auto full = [&](int n) { return warp_wait(bar(B_FULL + n % S), (uint32_t)(n / S) & 1u, s_abort); };
      bool ok = warp_wait(bar(B_KV), 0u, s_abort);
      // step i: S' and dP' of block i + 2 (i >= -2) behind dV and dK of block i, whose planes they overwrite
#pragma unroll 1
      for (int i = -2; i < nqb && ok; ++i) {
        if (i >= 0) {
          ok = warp_wait(bar(B_PREADY + (i & 1)), (uint32_t)(i >> 1) & 1u, s_abort);
          if (!ok) break;
          tc_fence_after();
          const uint32_t r = tmem + (uint32_t)(192 * (i & 1));
          mma_planes<NP>(tmem + T_DV, r, r + 128u, 32u, slot(2 * i), nv, i > 0);
          tc_commit(bar(B_FREE + (2 * i) % S));
          mma_planes<NP>(tmem + T_DK, r + 64u, r + 144u, 32u, slot(2 * i + 1), nd, i > 0);
          tc_commit(bar(B_FREE + (2 * i + 1) % S));
          if (i == nqb - 1) tc_commit(bar(B_DONE));
        }
        const int t = i + 2;
        if (t < nqb) {
          const uint32_t r = tmem + (uint32_t)(192 * (t & 1));
          ok = full(2 * t);
          if (!ok) break;
          tc_fence_after();
          mma_rows_s<NP>(r + 64u, sb + cfg::V_OFF, slot(2 * t));
          ok = full(2 * t + 1);
          if (!ok) break;
          tc_fence_after();
          mma_rows_s<NP>(r, sb + cfg::K_OFF, slot(2 * t + 1));
          tc_commit(bar(B_SFULL + (t & 1)));
        }
      }
    }
  } else {
    // ------------------------------------------------------------ compute warps ---
    const int set = (warp - 2) >> 2, qd = warp & 3;
    const int64_t kj = j0 + 32 * qd + lane;   // this thread's key
    const bool live = kj < D.Lk;
    const uint32_t t_row = tmem + ((uint32_t)(32 * qd) << 16);
    const int64_t el = NP == 3 ? 4 : 2;
    bool ok = true;
    for (int i = set; i < nqb && ok; i += 2) {
      const int n = 2 * i;
      ok = mbar_wait(bar(B_FULL + n % S), (uint32_t)(n / S) & 1u, s_abort) && mbar_wait(bar(B_SFULL + set), (uint32_t)(i >> 1) & 1u, s_abort);
      if (!ok) break;
      tc_fence_after();
      const float4* row = (const float4*)(cta.smem + (n % S) * cfg::SLOT_BYTES + NP * TILE);   // {lse, delta} of two queries
      // queries of the block this key is seen by: query < Lq (dead ones carry lse = inf), and query >= key when causal
      const int64_t i0b = (int64_t)(ib0 + i) * KT;
      int clo = 0;
      if (D.causal && kj - i0b > 0) clo = (kj - i0b) > KT ? KT : (int)(kj - i0b);
      if (!live) clo = KT;
      const uint32_t r = t_row + (uint32_t)(192 * set);
#pragma unroll
      for (int hf = 0; hf < 2; ++hf) {
        uint32_t sv[32], dp[32];
        tc_ld_32x32b_x32(r + 32u * hf, sv);
        tc_ld_32x32b_x32(r + 64u + 32u * hf, dp);
        tc_wait_ld();
#pragma unroll
        for (int c = 0; c < 32; c += 2) {
          const float4 w = row[16 * hf + (c >> 1)];
          float p0 = fast_exp2(fmaf(__uint_as_float(sv[c]), D.scale_log2, -w.x));
          float p1 = fast_exp2(fmaf(__uint_as_float(sv[c + 1]), D.scale_log2, -w.z));
          if (c + 32 * hf < clo) p0 = 0.0f;
          if (c + 1 + 32 * hf < clo) p1 = 0.0f;
          sv[c] = __float_as_uint(p0);
          sv[c + 1] = __float_as_uint(p1);
          dp[c] = __float_as_uint(p0 * (__uint_as_float(dp[c]) - w.y));
          dp[c + 1] = __float_as_uint(p1 * (__uint_as_float(dp[c + 1]) - w.w));
        }
        // over columns this thread has read already; the third planes lie behind both
        store_planes32(r + 32u * hf, r + 32u * hf + 16u, r + 128u + 32u * hf, sv);
        store_planes32(r + 64u + 32u * hf, r + 80u + 32u * hf, r + 144u + 32u * hf, dp);
      }
      tc_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar(B_PREADY + set));
    }
    // the first set writes dV, the second dK (scaled by 1 / sqrt(d)); zero where no query sees the keys
    if (ok && nqb > 0) ok = mbar_wait(bar(B_DONE), 0u, s_abort);
    if (ok) {
      tc_fence_after();
      uint8_t* drow = set == 0 ? (uint8_t*)dv + el * ((b * D.Lk + kj) * D.Ev + (int64_t)h * D.dv)
                               : (uint8_t*)dk + el * ((b * D.Lk + kj) * D.E + (int64_t)h * D.d);
#pragma unroll
      for (int hf = 0; hf < 2; ++hf) {
        uint32_t v[32];
        if (nqb > 0) {
          tc_ld_32x32b_x32(t_row + (set == 0 ? T_DV : T_DK) + 32u * hf, v);
          tc_wait_ld();
        } else {
#pragma unroll
          for (int c = 0; c < 32; ++c) v[c] = 0u;
        }
        if (live) store_row32<NP == 1>(drow, 32 * hf, set == 0 ? D.dv : D.d, D.vec != 0, (const float*)v, set == 0 ? 1.0f : D.scale);
      }
    }
  }
}

__global__ void __launch_bounds__(BWD_THREADS, 1)
attn_bwd_dkdv_tc_kernel(const uint8_t* __restrict__ qimg, const uint8_t* __restrict__ doimg, const uint8_t* __restrict__ kimg, const uint8_t* __restrict__ vimg,
                        const float2* __restrict__ rv, uint16_t* __restrict__ dk, uint16_t* __restrict__ dv, AtcDims D, int32_t* __restrict__ dev_err) {
  fb_after_previous();
  extern __shared__ uint8_t smem_raw[];
  Cta cta;
  if (!cta_begin(cta, smem_raw, KvCfg<1>::NOTES, 512u, dev_err, [](uint32_t sb) { KvCfg<1>::init(sb + KvCfg<1>::BAR); })) return;
  dkdv_item<1>(cta, cta.sb + KvCfg<1>::BAR, (int64_t)blockIdx.x * QT, (int)blockIdx.y, (int64_t)blockIdx.z, qimg, doimg, kimg, vimg, rv, dk, dv, D);
  cta_end(cta, 512u, dev_err, 4004);
}

// Float32 heads, picked ones: kv_items items of dK and dV, then those of dQ (each may be none)
__global__ void __launch_bounds__(BWD_THREADS, 1)
attn_bwd_picked_kernel(const float* __restrict__ q, const float* __restrict__ dout, const uint8_t* __restrict__ kimg, const uint8_t* __restrict__ vimg,
                       const uint8_t* __restrict__ qimg, const uint8_t* __restrict__ doimg, const float2* __restrict__ rv, float* __restrict__ dq,
                       float* __restrict__ dk, float* __restrict__ dv, const uint8_t* __restrict__ pick, int64_t kv_items, int64_t items, AtcDims D,
                       int32_t* __restrict__ dev_err) {
  fb_after_previous();
  fb_let_next_start();
  extern __shared__ uint8_t smem_raw[];
  const int64_t heads = kv_items > 0 ? kv_items / (D.ktiles / 2) : items / (D.qtiles / 2);
  auto head_of = [&](int64_t item) { return (item < kv_items ? item : item - kv_items) % heads; };
  const uint32_t mine = picked_items(pick, items, head_of);
  if (mine == 0) return;
  using kv = KvCfg<3>;
  using qc = DqCfg<3>;
  static_assert((int)qc::B_COUNT <= (int)kv::B_COUNT && qc::BAR <= kv::BAR, "one layout");
  auto bars = [](uint32_t sb, int n) { return sb + (uint32_t)(kv::BAR + 8 * kv::B_COUNT * n); };
  Cta cta;
  if (!cta_begin(cta, smem_raw, kv::NOTES, 512u, dev_err, [&](uint32_t sb) {
        for (int n = 0; n < PICK_ITEMS; ++n) {
          if (blockIdx.x + (int64_t)n * gridDim.x < kv_items) kv::init(bars(sb, n));
          else qc::init(bars(sb, n));
        }
      }))
    return;
  for (int n = 0; n < PICK_ITEMS; ++n) {
    if (!(mine >> n & 1)) continue;
    const int64_t item = blockIdx.x + (int64_t)n * gridDim.x, bh = head_of(item), b = bh / D.H;
    const int h = (int)(bh - b * D.H);
    if (item < kv_items) dkdv_item<3>(cta, bars(cta.sb, n), item / heads * QT, h, b, qimg, doimg, kimg, vimg, rv, dk, dv, D);
    else dq_item<3>(cta, bars(cta.sb, n), (D.qtiles / 2 - 1 - (item - kv_items) / heads) * QT, h, b, q, dout, kimg, vimg, rv, dq, D);
    if (!cta_next(cta)) break;
  }
  cta_end(cta, 512u, dev_err, 4004);
}

// CTAs for so many items: what the GPU holds at once, or more where a CTA would have more than PICK_ITEMS; an odd number beyond one item each, so that the
// tiles of a single head (items that lie the number of heads apart) are different CTAs'.
unsigned pick_grid(int64_t items, int64_t resident) {
  if (items <= resident) return (unsigned)items;
  const int64_t least = (items + PICK_ITEMS - 1) / PICK_ITEMS;
  return (unsigned)(least > resident ? least | 1 : (resident - 1) | 1);
}

// Heads with a value that is not finite are computed again by the FMA kernels.  Planes cannot carry one (the remainder of an infinite value
// is NaN, and so is an infinite plane times a zero one), while the sums of products give what such a value makes: a key of -inf no weight, a
// value of inf an infinite output.  The launch that finds nothing costs 4 - 6 us (2048 x 2048, 8 heads of 32, batch 2: 114 -> 119 us; the
// FMA kernel 853).
int32_t fwd_bf16(fb_ctx* ctx, cudaStream_t stream, const uint16_t* q, const uint16_t* k, const uint16_t* v, float* o, uint16_t* o16, float* lse,
                 const AtcPlan& P, int64_t batch) {
  const AtcDims& D = P.D;
  // a byte for every K and V tile and every 32 queries of a (batch, head)
  const int odd_n = 2 * D.ktiles + 2 * D.qtiles;
  const int64_t per = 2 * P.kbytes + (int64_t)D.H * odd_n;
  int64_t chunk = IMAGE_BYTES / per;
  chunk = chunk < 1 ? 1 : (chunk > batch ? batch : chunk);
  const fb_temp images(ctx, stream, (size_t)(chunk * per));
  uint8_t* img = (uint8_t*)images.p;
  if (!img) return FB_ERR_UNSUPPORTED;
  FB_ONCE(ctx, FB_CUDA(cudaFuncSetAttribute(attn_fwd_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, FwdCfg<1>::SMEM)));
  for (int64_t b0 = 0; b0 < batch; b0 += chunk) {
    const int64_t nb = b0 + chunk > batch ? batch - b0 : chunk;
    uint8_t* odd = img + nb * 2 * P.kbytes;
    const uint16_t *qb = q + b0 * D.Lq * D.E, *kb = k + b0 * D.Lk * D.E, *vb = v + b0 * D.Lk * D.Ev;
    float *ob = o ? o + b0 * D.Lq * D.Ev : nullptr, *lb = lse + b0 * D.H * D.Lq;
    uint16_t* ob16 = o16 + b0 * D.Lq * D.Ev;
    SplitArgs A = {};
    A.H = D.H; A.vec = D.vec; A.odd = odd; A.odd_n = odd_n; A.max_tiles = D.ktiles;
    A.job[0] = {kb, img, D.Lk, D.E, D.d, D.ktiles};
    A.job[1] = {vb, img + nb * P.kbytes, D.Lk, D.Ev, D.dv, D.ktiles};
    fb_launch(attn_split_kernel, dim3((unsigned)D.ktiles, (unsigned)(nb * D.H), 2), 256, 0, stream, A);
    FB_LAUNCH_CHECK();
    fb_launch(attn_fwd_tc_kernel, dim3((unsigned)(D.qtiles / 2), (unsigned)D.H, (unsigned)nb), FWD_THREADS, FwdCfg<1>::SMEM, stream, qb, img, img + nb * P.kbytes, ob, ob16, lb,
              odd + 2 * D.ktiles, odd_n, D, ctx->dev_error);
    FB_LAUNCH_CHECK();
    const int32_t st = fb_attn_fwd_redo(ctx, stream, 1, qb, kb, vb, ob, ob16, lb, D.E, D.Ev, D.Lq, D.Lk, nb, D.H, D.causal, odd, odd_n);
    if (st != FB_OK) return st;
  }
  return FB_OK;
}

int32_t bwd_bf16(fb_ctx* ctx, cudaStream_t stream, const uint16_t* q, const uint16_t* k, const uint16_t* v, const float* o, const float* lse, const uint16_t* dout,
                 uint16_t* dq, uint16_t* dk, uint16_t* dv, const AtcPlan& P, int64_t batch) {
  const AtcDims& D = P.D;
  const int odd_n = 4 * D.max_tiles;   // a byte for every tile of a (batch, head)
  const int64_t per = 2 * P.kbytes + 2 * P.qbytes + P.rvbytes + (int64_t)D.H * odd_n;
  int64_t chunk = IMAGE_BYTES / per;
  chunk = chunk < 1 ? 1 : (chunk > batch ? batch : chunk);
  const fb_temp images(ctx, stream, (size_t)(chunk * per));
  uint8_t* img = (uint8_t*)images.p;
  if (!img) return FB_ERR_UNSUPPORTED;
  FB_ONCE(ctx, FB_CUDA(cudaFuncSetAttribute(attn_bwd_dkdv_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, KvCfg<1>::SMEM)));
  FB_ONCE(ctx, FB_CUDA(cudaFuncSetAttribute(attn_bwd_dq_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, DqCfg<1>::SMEM)));
  for (int64_t b0 = 0; b0 < batch; b0 += chunk) {
    const int64_t nb = b0 + chunk > batch ? batch - b0 : chunk;
    uint8_t *ki = img, *vi = ki + nb * P.kbytes, *qi = vi + nb * P.kbytes, *doi = qi + nb * P.qbytes;
    float2* rv = (float2*)(doi + nb * P.qbytes);
    uint8_t* odd = (uint8_t*)rv + nb * P.rvbytes;
    const int64_t qoff = b0 * D.Lq * D.E, qvoff = b0 * D.Lq * D.Ev, koff = b0 * D.Lk * D.E, kvoff = b0 * D.Lk * D.Ev;
    const uint16_t *qb = q + qoff, *kb = k + koff, *vb = v + kvoff, *dob = dout + qvoff;
    const float* lb = lse + b0 * D.H * D.Lq;
    SplitArgs A = {};
    A.H = D.H; A.vec = D.vec; A.odd = odd; A.odd_n = odd_n; A.max_tiles = D.max_tiles;
    A.job[0] = {kb, ki, D.Lk, D.E, D.d, D.ktiles};
    A.job[1] = {vb, vi, D.Lk, D.Ev, D.dv, D.ktiles};
    A.job[2] = {qb, qi, D.Lq, D.E, D.d, D.qtiles};
    A.job[3] = {dob, doi, D.Lq, D.Ev, D.dv, D.qtiles};
    A.o = o + qvoff; A.lse = lb; A.rv = rv;
    // (tiles that one operand has and another has not keep no byte)
    if (D.qtiles != D.ktiles) FB_CUDA(cudaMemsetAsync(odd, 0, (size_t)(nb * D.H * odd_n), stream));
    fb_launch(attn_split_kernel, dim3((unsigned)D.max_tiles, (unsigned)(nb * D.H), 4), 256, 0, stream, A);
    FB_LAUNCH_CHECK();
    fb_launch(attn_bwd_dkdv_tc_kernel, dim3((unsigned)(D.ktiles / 2), (unsigned)D.H, (unsigned)nb), BWD_THREADS, KvCfg<1>::SMEM, stream, qi, doi, ki, vi, rv, dk + koff,
              dv + kvoff, D, ctx->dev_error);
    FB_LAUNCH_CHECK();
    fb_launch(attn_bwd_dq_tc_kernel, dim3((unsigned)(D.qtiles / 2), (unsigned)D.H, (unsigned)nb), BWD_THREADS, DqCfg<1>::SMEM, stream, qb, dob, ki, vi, rv, dq + qoff, D,
              ctx->dev_error);
    FB_LAUNCH_CHECK();
    const int32_t st = fb_attn_bwd_redo(ctx, stream, 1, qb, kb, vb, lb, (const float*)rv + 1, (int64_t)D.qtiles * KT, dob, dq + qoff, dk + koff, dv + kvoff, D.E, D.Ev,
                                        D.Lq, D.Lk, nb, D.H, D.causal, odd, odd_n);
    if (st != FB_OK) return st;
  }
  return FB_OK;
}

}  // namespace

int32_t fb_atc::fwd_picked(fb_ctx* ctx, cudaStream_t stream, const float* q, const uint8_t* kimg, const uint8_t* vimg, float* o, float* lse, const AtcDims& D, int64_t batch,
                           const uint8_t* pick) {
  FB_ONCE(ctx, FB_CUDA(cudaFuncSetAttribute(attn_fwd_picked_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, FwdCfg<3>::SMEM)));
  const int64_t items = batch * D.H * (D.qtiles / 2);
  fb_launch(attn_fwd_picked_kernel, pick_grid(items, 2 * (int64_t)ctx->sm_count), FWD_THREADS, FwdCfg<3>::SMEM, stream, q, kimg, vimg, o, lse, pick, items, D, ctx->dev_error);
  FB_LAUNCH_CHECK();
  return FB_OK;
}

int32_t fb_atc::bwd_picked(fb_ctx* ctx, cudaStream_t stream, const float* q, const float* dout, const uint8_t* kimg, const uint8_t* vimg, const uint8_t* qimg,
                           const uint8_t* doimg, const float2* rv, float* dq, float* dk, float* dv, const AtcDims& D, int64_t batch, const uint8_t* pick) {
  FB_ONCE(ctx, FB_CUDA(cudaFuncSetAttribute(attn_bwd_picked_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, KvCfg<3>::SMEM)));
  const int64_t kv_items = dk != nullptr ? batch * D.H * (D.ktiles / 2) : 0, items = kv_items + (dq != nullptr ? batch * D.H * (D.qtiles / 2) : 0);
  fb_launch(attn_bwd_picked_kernel, pick_grid(items, ctx->sm_count), BWD_THREADS, KvCfg<3>::SMEM, stream, q, dout, kimg, vimg, qimg, doimg, rv, dq, dk, dv, pick, kv_items,
            items, D, ctx->dev_error);
  FB_LAUNCH_CHECK();
  return FB_OK;
}

// bf16 q, k, v (and dO): one plane each, outputs rounded to bf16 once.  o32 (optional in the forward call) keeps
// the Float32 output for the backward pass.  FB_ERR_UNSUPPORTED, without a message, for every call these kernels do not
// take: the caller then casts and takes the Float32 entry points, which also report what is wrong with a bad one.  The
// backward call takes the head size of the Float32 one, for the same reason.
FB_API int32_t fb_attn_fwd_bf16(fb_ctx* ctx, void* stream, const uint16_t* q, const uint16_t* k, const uint16_t* v, float* o32, uint16_t* o,
                                float* lse, int64_t e_dim, int64_t ev_dim, int64_t lq, int64_t lk, int64_t batch, int32_t nheads,
                                int32_t causal) {
  FB_CHECK_CTX(ctx);
  AtcPlan P;
  if (!attn_tc_enabled() || !q || !k || !v || !o || !lse || nheads < 1 || e_dim % nheads != 0 || ev_dim % nheads != 0 || batch * nheads > 65535 ||
      !make_plan(&P, 1, e_dim, ev_dim, lq, lk, batch, nheads, causal))
    return FB_ERR_UNSUPPORTED;
  if (!fb_aligned16(q) || !fb_aligned16(k) || !fb_aligned16(v) || !fb_aligned16(o) || !fb_aligned16(o32)) return FB_ERR_UNSUPPORTED;
  return fwd_bf16(ctx, (cudaStream_t)stream, q, k, v, o32, o, lse, P, batch);
}

FB_API int32_t fb_attn_bwd_bf16(fb_ctx* ctx, void* stream, const uint16_t* q, const uint16_t* k, const uint16_t* v, const float* o32,
                                const float* lse, const uint16_t* dout, uint16_t* dq, uint16_t* dk, uint16_t* dv, int64_t e_dim, int64_t ev_dim,
                                int64_t lq, int64_t lk, int64_t batch, int32_t nheads, int32_t causal) {
  FB_CHECK_CTX(ctx);
  AtcPlan P;
  if (!attn_tc_enabled() || !attn_bwd_tc_enabled() || !q || !k || !v || !o32 || !lse || !dout || !dq || !dk || !dv || nheads < 1 ||
      e_dim % nheads != 0 || ev_dim % nheads != 0 || batch * nheads > 65535 || lq > BWD_MAX_BLOCKS * KT || lk > BWD_MAX_BLOCKS * KT ||
      !make_plan(&P, 1, e_dim, ev_dim, lq, lk, batch, nheads, causal) || P.D.d != HD || P.D.dv != HD)
    return FB_ERR_UNSUPPORTED;
  if (!fb_aligned16(q) || !fb_aligned16(k) || !fb_aligned16(v) || !fb_aligned16(o32) || !fb_aligned16(dout) || !fb_aligned16(dq) ||
      !fb_aligned16(dk) || !fb_aligned16(dv))
    return FB_ERR_UNSUPPORTED;
  return bwd_bf16(ctx, (cudaStream_t)stream, q, k, v, o32, lse, dout, dq, dk, dv, P, batch);
}
