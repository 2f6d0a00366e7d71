// Flash-style attention of Float32 operands on the tensor cores (tcgen05), for head sizes up to 64 forward and of 64 backward.
//
// An operand is two half-precision planes, x 2^s = hi + lo 2^-11 (23 bits; a power of two per tile or row), and a product is the
// sum of three plane products: the cross terms first, then hi hi over 2^-11 of them (the MMA scales its accumulator), or, where
// sums go on over the blocks, in accumulators of their own.  An image in the 128-byte swizzle serves as K-major and as MN-major operand;
// a small kernel (`attn_half_split_kernel`) makes the images of K, V, Q and dO once per call, and tiles arrive by plain bulk copies.
// Head sizes below 64 are padded with zeros in the images; their zero 16-feature steps are skipped.
//
// Against three bf16 planes per operand and six products (batch 8, 16 heads of 64, 2048 x 2048, causal; us): forward 507 -> 349, dK / dV 1113 -> 618,
// dQ 848 -> 503; images 51 + 114 -> 67 + 104 (with a look at Q ahead of the forward kernel).  Errors against float64: output 2.3e-7
// as before, dQ 4.7e-6 -> 0.9e-6, dK / dV 1.9e-5 -> 3.8e-6 (half as many truncating adds).  Heads that these planes would hold worse are left to
// attention_tc.cu, see below.
// What bounds them: an MMA with N = 64 takes 53 clocks with A in tensor memory and 74 with A in shared memory, where its multiplications
// need 32, and between the MMAs of a block the weights' arithmetic (one warp of a set per SM partition, 3700 clocks a block).
//
// A block is 64 keys (64 queries in the dK / dV kernel) against the 128 rows of a CTA; a thread of a compute warp owns
// one row (one TMEM lane).  Every mbarrier wait is bounded; when one runs out the kernel records 4002 (forward), 4003
// (dQ) or 4004 (dK / dV) in the context's device error word, all roles leave their loops, tensor memory is released and
// the kernel returns.
#include <cuda_fp16.h>

#include "attention_tc.cuh"

using namespace fb_atc;

namespace {

constexpr int NP = 2;             // planes of an operand
constexpr int SLOT = 3 * TILE;    // memory of a tile's images: these two planes, or the three bf16 ones of a head that is left to attention_tc.cu

// the same where D is first multiplied by 2^-11 (A from tensor memory; A from shared memory)
__device__ __forceinline__ void tc_mma_ta_down(uint32_t d_tmem, uint32_t a_tmem, uint32_t b_lo, uint32_t hi, uint32_t idesc) {
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t.reg .b64 db;\n\t"
      "elect.sync _|q, 0xffffffff;\n\t"
      "setp.eq.b32 p, %4, 0;\n\t"
      "mov.b64 db, {%2, %5};\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], db, %3, {%4, %4, %4, %4}, p, 11;\n\t}"
      ::"r"(d_tmem), "r"(a_tmem), "r"(b_lo), "r"(idesc), "r"(0u), "r"(hi)
      : "memory");
}
__device__ __forceinline__ void tc_mma_sa_down(uint32_t d_tmem, uint32_t a_lo, uint32_t b_lo, uint32_t hi, uint32_t idesc) {
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t.reg .b64 da, db;\n\t"
      "elect.sync _|q, 0xffffffff;\n\t"
      "setp.eq.b32 p, %4, 0;\n\t"
      "mov.b64 da, {%1, %5};\n\t"
      "mov.b64 db, {%2, %5};\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %3, {%4, %4, %4, %4}, p, 11;\n\t}"
      ::"r"(d_tmem), "r"(a_lo), "r"(b_lo), "r"(idesc), "r"(0u), "r"(hi)
      : "memory");
}
// Two values as two half-precision planes (x in the low half of each word): the upper one rounded to nearest, the lower one the
// remainder times 2^11, so that it keeps its bits as long as the upper one does.
__device__ __forceinline__ void split2(float x, float y, uint32_t& hi, uint32_t& lo) {
  const __half2 h = __floats2half2_rn(x, y);
  const float2 f = __half22float2(h);
  const __half2 l = __floats2half2_rn((x - f.x) * 2048.0f, (y - f.y) * 2048.0f);
  hi = *reinterpret_cast<const uint32_t*>(&h);
  lo = *reinterpret_cast<const uint32_t*>(&l);
}
// Scales are powers of two, as shifts: 2^s puts a largest magnitude (its bits) into [2^14, 2^15).  What is scaled so is held to 2^-23
// of itself down to 2^-29 of the largest value and to 2^-51 of that below.  Three bf16 planes hold 2^-24 at any exponent, so a head is
// left to them ("picked") where that would show:
// - scores that may exceed SCORE_LIMIT, by the row norms of Q and K.  An exponential turns a relative error into an absolute one, and weights below
//   2^-29 lose bits.  Heads of 512 x 512 with scores of standard deviation 1, 2, 4, 8, 16 (largest bound 16, 31, 62, ...): errors of the output
//   2.1, 3.4, 3.5, 4.5, 5.7e-7 here and 2.1, 3.3, 3.2, 3.8, 4.8e-7 with three planes, of dQ 0.4 - 2.3e-6 and 1.4 - 2.6e-6; one key and one value
//   1e4 times the others: output 3.6e-6 and 6.2e-7, dQ 4.3e-3 and 1.6e-4.
// - a tile with a row or a column (of the operand: a position or a feature) whose largest value is below 2^-19 of the tile's.  So a value
//   is held to 2^-23 of itself or to 2^-32 of the largest of its row and of its column.
// - backward, tiles whose scales differ by more than 2^SH_SPREAD: dS is made in one unit for the head.
// - values out of the range of the scales.
// Heads with a value that is not finite are the FMA kernels'.
constexpr int SH_ZERO = 1000;    // all values are 0
__device__ __forceinline__ int shift_of(uint32_t max_bits) { return max_bits == 0 ? SH_ZERO : 141 - (int)(max_bits >> 23); }
__device__ __forceinline__ float pow2(int e) { return e < -126 ? 0.0f : __int_as_float((e > 127 ? 254 : e + 127) << 23); }
// v 2^e in two factors, |e| <= 252
__device__ __forceinline__ float times_pow2(float v, int e) {
  const int h = e / 2;
  return v * pow2(h) * pow2(e - h);
}
constexpr uint32_t FAINT_BITS = 19u << 23;   // 2^-19, as what the bits of a magnitude differ by
constexpr float SCORE_LIMIT = 32.0f;
// largest shifts, up or down, of Q and K, of V and of dO: products of two of their powers of two stay in range
constexpr int SH_QK = 60, SH_V = 40, SH_DO = 85;

// 32 values of a thread's row into the two planes of an A operand: 16 columns each at t0 and t1
__device__ __forceinline__ void store_planes32(uint32_t t0, uint32_t t1, const uint32_t* v) {
  uint32_t a[16], b[16];
#pragma unroll
  for (int e = 0; e < 16; ++e) split2(__uint_as_float(v[2 * e]), __uint_as_float(v[2 * e + 1]), a[e], b[e]);
  tc_st_32x32b_x16(t0, a);
  tc_st_32x32b_x16(t1, b);
}

// One row of a CTA's own operand into tensor memory: planes of 32 columns each, scaled by 2^sh.
__device__ __forceinline__ void row_to_tmem(const void* src, int width, bool live, bool vec, uint32_t t_addr, int limit, int& sh) {
  uint32_t v[2][32];
#pragma unroll
  for (int hf = 0; hf < 2; ++hf) row_f32((const float*)src, 32 * hf, width, live, vec, v[hf]);
  uint32_t m = 0u;
#pragma unroll
  for (int c = 0; c < 64; ++c) m = max(m, v[c >> 5][c & 31] & 0x7fffffffu);
  sh = shift_of(m);
  sh = sh == SH_ZERO ? 0 : min(sh, limit);   // (not below -limit: the head would be picked)
  const float sc = pow2(sh);
#pragma unroll
  for (int hf = 0; hf < 2; ++hf) {
#pragma unroll
    for (int c = 0; c < 32; ++c) v[hf][c] = __float_as_uint(__uint_as_float(v[hf][c]) * sc);
    store_planes32(t_addr + 16u * hf, t_addr + 32u + 16u * hf, v[hf]);
  }
}

// instruction descriptors: D = F32, A = B = F16, M = 128; B K-major (n columns = rows of the tile) or MN-major
__device__ __forceinline__ uint32_t idesc_f16(int n, bool b_mn) {
  return (1u << 4) | ((b_mn ? 1u : 0u) << 16) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(QT >> 4) << 24);
}
// The plane products: the cross terms (2^11 too large), then the product of the upper planes over the sum of those times 2^-11.  (The
// product of the lower planes is below 2^-24 of the whole.)
//
// D = A B', A = planes in tensor memory (32 columns each), B = K-major planes; nks steps of 16 features
__device__ __forceinline__ void mma_rows_t(uint32_t d, uint32_t a_tmem, uint32_t b_smem, int nks) {
  const uint64_t b0 = desc_k(b_smem);
  const uint32_t idesc = idesc_f16(KT, false), hi = (uint32_t)(b0 >> 32), b = (uint32_t)b0;
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int ks = 0; ks < 4; ++ks)
      if (ks < nks)
        tc_mma_ta(d, a_tmem + (uint32_t)(32 * (1 - i) + 8 * ks), b + (uint32_t)((i * TILE + ks * 32) >> 4), hi, idesc, (i > 0 || ks > 0) ? 1u : 0u);
#pragma unroll
  for (int ks = 0; ks < 4; ++ks)
    if (ks < nks) {
      if (ks == 0) tc_mma_ta_down(d, a_tmem, b, hi, idesc);
      else tc_mma_ta(d, a_tmem + (uint32_t)(8 * ks), b + (uint32_t)((ks * 32) >> 4), hi, idesc, ks > 0 ? 1u : 0u);
    }
}
// the same with A in shared memory: planes of 128 rows, 2 * TILE apart, all four steps (head sizes are zero-padded)
__device__ __forceinline__ void mma_rows_s(uint32_t d, uint32_t a_smem, uint32_t b_smem) {
  const uint64_t a0 = desc_k(a_smem), b0 = desc_k(b_smem);
  const uint32_t idesc = idesc_f16(KT, false), hi = (uint32_t)(a0 >> 32), a = (uint32_t)a0, b = (uint32_t)b0;
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int ks = 0; ks < 4; ++ks)
      tc_mma_sa(d, a + (uint32_t)(((1 - i) * 2 * TILE + ks * 32) >> 4), b + (uint32_t)((i * TILE + ks * 32) >> 4), hi, idesc, (i > 0 || ks > 0) ? 1u : 0u);
#pragma unroll
  for (int ks = 0; ks < 4; ++ks) {
    if (ks == 0) tc_mma_sa_down(d, a, b, hi, idesc);
    else tc_mma_sa(d, a + (uint32_t)((ks * 32) >> 4), b + (uint32_t)((ks * 32) >> 4), hi, idesc, ks > 0 ? 1u : 0u);
  }
}
// A = two planes of 64 values in tensor memory that the compute warps stored in halves of 32 values (the upper plane at t + 32 half,
// the lower one sixteen columns behind it), B = MN-major planes whose K rows are the tile's rows; n columns (features, a multiple
// of 16).  D = A B; or, with sums that go on over the blocks, D += upper A upper B and X += the cross terms, 2^11 too large.
__device__ __forceinline__ uint32_t plane_step(uint32_t t, int lower, int ks) { return t + (uint32_t)(32 * (ks >> 1) + 16 * lower + 8 * (ks & 1)); }
__device__ __forceinline__ void mma_planes(uint32_t d, uint32_t t, uint32_t b_smem, int n) {
  const uint64_t b0 = desc_mn(b_smem);
  const uint32_t idesc = idesc_f16(n, true), hi = (uint32_t)(b0 >> 32), b = (uint32_t)b0;
#pragma unroll
  for (int i = 0; i < NP; ++i)
#pragma unroll
    for (int ks = 0; ks < 4; ++ks)
      tc_mma_ta(d, plane_step(t, 1 - i, ks), b + (uint32_t)((i * TILE + ks * 2048) >> 4), hi, idesc, (i > 0 || ks > 0) ? 1u : 0u);
#pragma unroll
  for (int ks = 0; ks < 4; ++ks) {
    if (ks == 0) tc_mma_ta_down(d, plane_step(t, 0, 0), b, hi, idesc);
    else tc_mma_ta(d, plane_step(t, 0, ks), b + (uint32_t)((ks * 2048) >> 4), hi, idesc, 1u);
  }
}
__device__ __forceinline__ void mma_planes_sum(uint32_t d, uint32_t x, uint32_t t, uint32_t b_smem, int n, bool go_on) {
  const uint64_t b0 = desc_mn(b_smem);
  const uint32_t idesc = idesc_f16(n, true), hi = (uint32_t)(b0 >> 32), b = (uint32_t)b0;
#pragma unroll
  for (int i = 0; i < NP; ++i)
#pragma unroll
    for (int ks = 0; ks < 4; ++ks)
      tc_mma_ta(x, plane_step(t, 1 - i, ks), b + (uint32_t)((i * TILE + ks * 2048) >> 4), hi, idesc, (go_on || i > 0 || ks > 0) ? 1u : 0u);
#pragma unroll
  for (int ks = 0; ks < 4; ++ks)
    tc_mma_ta(d, plane_step(t, 0, ks), b + (uint32_t)((ks * 2048) >> 4), hi, idesc, (go_on || ks > 0) ? 1u : 0u);
}

// -------------------------------------------------------------------------------------------- plane images ---
// One 64 x 64 tile of one (batch, head): rows scaled by a power of two per tile -> two half-precision planes, each
// the shared-memory image of the tile (row r at 128 r, its 16-byte chunks permuted by r & 7); rows past the end and features past
// the head size are 0.  For dO the same pass forms what the softmax backward needs per query: {log2(e) lse, delta = sum_c dO_c O_c};
// queries past the end get {inf, 0}, which makes their weights 0.
// The notes say what the tile is like.  A job without images (Q ahead of the forward kernel) only gets those.
// Bound by memory: 4 bytes in, 4 out per value.
struct TileNote {
  float norm2;      // largest squared norm of a row
  int16_t shift;
  int16_t odd;      // 1: the planes do not hold the tile well, 2: a value is not finite
};
struct SplitJob {
  const void* src;
  uint8_t* dst;
  int64_t L, E;
  int width, tiles, limit;
};
struct SplitArgs {
  SplitJob job[4];
  const float* o;       // for the job of index 3 (dO)
  const float* lse;
  float2* rv;
  TileNote* notes;      // [batch head][job][max_tiles]
  int H, vec, jobs, max_tiles;
};

constexpr int SPLIT_THREADS = KT * 8, SPLIT_WARPS = SPLIT_THREADS / 32;   // eight values of a row a thread (sixteen of two rows: 78 us for 134 MB of Q, K and V, here 67)
__global__ void __launch_bounds__(SPLIT_THREADS, 4) attn_half_split_kernel(SplitArgs A) {
  fb_after_previous();
  __shared__ uint32_t top[SPLIT_WARPS];
  __shared__ float norms[SPLIT_WARPS];
  __shared__ uint32_t cols[SPLIT_WARPS][KT];
  const SplitJob J = A.job[blockIdx.z];
  if ((int)blockIdx.x >= J.tiles) return;
  const int64_t bh = blockIdx.y;
  const int64_t b = bh / A.H;
  const int h = (int)(bh - b * A.H);
  const int r = threadIdx.x >> 3, ch = threadIdx.x & 7;
  const int64_t row = (int64_t)blockIdx.x * KT + r;
  const bool live = row < J.L;
  const int64_t off = (b * J.L + row) * J.E + (int64_t)h * J.width;
  const float* src = (const float*)J.src + off;
  float x[8];
  if (A.vec) {
#pragma unroll
    for (int e = 0; e < 8; e += 4) {
      float4 t = make_float4(0.f, 0.f, 0.f, 0.f);
      if (live && 8 * ch + e < J.width) t = __ldg((const float4*)(src + 8 * ch + e));
      x[e] = t.x; x[e + 1] = t.y; x[e + 2] = t.z; x[e + 3] = t.w;
    }
  } else {
#pragma unroll
    for (int e = 0; e < 8; ++e) x[e] = (live && 8 * ch + e < J.width) ? __ldg(src + 8 * ch + e) : 0.0f;
  }
  if (blockIdx.z == 3) {   // dO
    float sum = 0.0f;
#pragma unroll
    for (int e = 0; e < 8; e += 4) {
      if (!live || 8 * ch + e >= J.width) break;
      const float* po = A.o + off + 8 * ch + e;
      if (A.vec) {
        const float4 t = __ldg((const float4*)po);
        sum = fmaf(x[e], t.x, sum); sum = fmaf(x[e + 1], t.y, sum); sum = fmaf(x[e + 2], t.z, sum); sum = fmaf(x[e + 3], t.w, sum);
      } else {
        for (int u = 0; u < 4 && 8 * ch + e + u < J.width; ++u) sum = fmaf(x[e + u], __ldg(po + u), sum);
      }
    }
    sum += __shfl_xor_sync(0xffffffffu, sum, 1);
    sum += __shfl_xor_sync(0xffffffffu, sum, 2);
    sum += __shfl_xor_sync(0xffffffffu, sum, 4);
    if (ch == 0) A.rv[bh * ((int64_t)J.tiles * KT) + row] = live ? make_float2(A.lse[bh * J.L + row] * LOG2E, sum) : make_float2(INFINITY, 0.0f);
  }
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  uint32_t m = 0u, least = ~0u;   // the largest magnitude, the least one that is not 0 (less 1)
#pragma unroll
  for (int e = 0; e < 8; ++e) {
    const uint32_t a = __float_as_uint(x[e]) & 0x7fffffffu;
    m = max(m, a);
    least = min(least, a - 1u);
  }
  const uint32_t own = m;   // the largest of this thread's eight
  m = __reduce_max_sync(0xffffffffu, m);
  float norm2 = 0.0f;
  if ((blockIdx.z & 1) == 0) {   // K and Q
#pragma unroll
    for (int e = 0; e < 8; ++e) norm2 = fmaf(x[e], x[e], norm2);
    norm2 += __shfl_xor_sync(0xffffffffu, norm2, 1);
    norm2 += __shfl_xor_sync(0xffffffffu, norm2, 2);
    norm2 += __shfl_xor_sync(0xffffffffu, norm2, 4);
    norm2 = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(norm2)));   // (not negative: the order is that of the bits)
  }
  if (lane == 0) {
    top[warp] = m;
    norms[warp] = norm2;
  }
  __syncthreads();
  m = __reduce_max_sync(0xffffffffu, top[lane % SPLIT_WARPS]);
  const int sh = shift_of(m);
  const bool in_range = sh == SH_ZERO || (sh <= J.limit && sh >= -J.limit);
  // (few tiles hold a value below the line at all: one of a hundred of normally distributed ones)
  const uint32_t line = m > FAINT_BITS ? m - FAINT_BITS : 0u;
  const bool look = __syncthreads_or(least != ~0u && least + 1u < line) != 0;
  if (J.dst != nullptr) {
    const float sc = pow2(sh == SH_ZERO || !in_range ? 0 : sh);
    uint8_t* out = J.dst + (bh * J.tiles + blockIdx.x) * (int64_t)SLOT + r * 128 + ((ch ^ (r & 7)) << 4);
    uint32_t p0[4], p1[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) split2(x[2 * e] * sc, x[2 * e + 1] * sc, p0[e], p1[e]);
    *(uint4*)out = make_uint4(p0[0], p0[1], p0[2], p0[3]);
    *(uint4*)(out + TILE) = make_uint4(p1[0], p1[1], p1[2], p1[3]);
  }
  bool faint = false;
  if (look) {
    uint32_t rmax = own;
#pragma unroll
    for (int o = 1; o < 8; o *= 2) rmax = max(rmax, __shfl_xor_sync(0xffffffffu, rmax, o));
    faint = rmax != 0u && rmax < line;
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      uint32_t col = __float_as_uint(x[e]) & 0x7fffffffu;
      col = max(col, __shfl_xor_sync(0xffffffffu, col, 8));
      col = max(col, __shfl_xor_sync(0xffffffffu, col, 16));
      if (lane < 8) cols[warp][8 * lane + e] = col;
    }
    __syncthreads();
    if (threadIdx.x < KT) {
      uint32_t col = 0u;
#pragma unroll 4
      for (int w = 0; w < SPLIT_WARPS; ++w) col = max(col, cols[w][threadIdx.x]);
      faint |= col != 0u && col < line;
    }
    faint = __syncthreads_or(faint) != 0;
  }
  if (threadIdx.x == 0) {
    for (int w = 1; w < SPLIT_WARPS; ++w) norm2 = fmaxf(norm2, norms[w]);
    TileNote note;
    note.norm2 = norm2;
    note.shift = (int16_t)sh;
    note.odd = (int16_t)(not_finite(m) ? 2 : faint || !in_range ? 1 : 0);
    A.notes[(bh * A.jobs + (int)blockIdx.z) * A.max_tiles + (int)blockIdx.x] = note;
  }
}

// How a head is computed: 0 here, 1 by attention_tc.cu, 2 by the FMA kernels.
struct HeadState {
  uint32_t odd, q, k;   // over its tiles: the largest note, the largest row norms (bits of the squares)
  __device__ __forceinline__ void add(int job, uint2 note) {
    if (note.y >> 16 != 0u) atomicMax(&odd, note.y >> 16);
    if (job == 0) atomicMax(&k, note.x);
    if (job == 2) atomicMax(&q, note.x);
  }
  __device__ __forceinline__ int state(const AtcDims& D) const {
    if (odd != 0u) return (int)odd;
    const float bound = sqrtf(__uint_as_float(q)) * sqrtf(__uint_as_float(k)) * D.scale;
    return bound <= SCORE_LIMIT ? 0 : 1;   // (also where a square has left the range)
  }
};
// The same for the forward kernel.  All threads; ends with a barrier.
__device__ __forceinline__ int head_state(HeadState& S, const TileNote* notes, const AtcDims& D) {
  if (threadIdx.x == 0) S = HeadState{0u, 0u, 0u};
  __syncthreads();
  for (int i = threadIdx.x; i < 3 * D.max_tiles; i += (int)blockDim.x) {
    const int job = i / D.max_tiles;
    if (i - job * D.max_tiles < (job < 2 ? D.ktiles : D.qtiles)) S.add(job, __ldg((const uint2*)(notes + i)));
  }
  __syncthreads();
  return S.state(D);
}
// The images of a picked head: three bf16 planes a tile, in the place of the planes here.  CTA `part` of the `parts` of the head takes its share of the tiles.
__device__ __noinline__ void images_of_three(const SplitArgs& A, int64_t bh, int part, int parts) {
  constexpr int U = 4;   // pieces of eight values on their way at once
  const int64_t b = bh / A.H;
  const int h = (int)(bh - b * A.H);
  for (int job = 0; job < A.jobs; ++job) {
    const SplitJob J = A.job[job];
    if (J.dst == nullptr) continue;
    const float* src = (const float*)J.src + b * J.L * J.E + (int64_t)h * J.width;
    const int own = (J.tiles - part + parts - 1) / parts * (KT * 8);   // pieces of this CTA's tiles part, part + parts, ...
    for (int i0 = threadIdx.x; i0 < own; i0 += U * (int)blockDim.x) {
      float x[U][8];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int i = i0 + u * (int)blockDim.x, ch = i & 7;
        const int64_t row = (int64_t)(part + (i >> 9) * parts) * KT + (i >> 3 & (KT - 1));
        const bool live = i < own && row < J.L;
        const float* p = src + row * J.E + 8 * ch;
        if (A.vec) {
#pragma unroll
          for (int e = 0; e < 8; e += 4) {
            float4 t = make_float4(0.f, 0.f, 0.f, 0.f);
            if (live && 8 * ch + e < J.width) t = __ldg((const float4*)(p + e));
            x[u][e] = t.x; x[u][e + 1] = t.y; x[u][e + 2] = t.z; x[u][e + 3] = t.w;
          }
        } else {
#pragma unroll
          for (int e = 0; e < 8; ++e) x[u][e] = (live && 8 * ch + e < J.width) ? __ldg(p + e) : 0.0f;
        }
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int i = i0 + u * (int)blockDim.x, ch = i & 7, r = i >> 3 & (KT - 1);
        if (i >= own) break;
        uint8_t* out = J.dst + (bh * J.tiles + part + (i >> 9) * parts) * (int64_t)SLOT + r * 128 + ((ch ^ (r & 7)) << 4);
        uint32_t q[3][4];
#pragma unroll
        for (int e = 0; e < 4; ++e) split3(x[u][2 * e], x[u][2 * e + 1], q[0][e], q[1][e], q[2][e]);
#pragma unroll
        for (int n = 0; n < 3; ++n) *(uint4*)(out + n * TILE) = make_uint4(q[n][0], q[n][1], q[n][2], q[n][3]);
      }
    }
  }
}
static_assert(KT * 8 == 512, "pieces of a tile");

// ------------------------------------------------------------------------------------------------------ forward ---
// One CTA owns 128 queries of one (batch, head); warp 0 copies K and V tiles into a ring of slots (K0 V0 K1 V1 ...),
// warp 1 issues the MMAs, warps 2-5 are the softmax (thread = query).  S = Q K' lands in 64 columns, the weights replace it
// as two planes, P V lands in 64 more columns and is added to the thread's registers with round-to-nearest adds.
// Within a CTA these steps follow one another; what keeps the tensor pipe busy is the SECOND CTA on the SM: 256 of the 512
// TMEM columns, half of the registers and of shared memory each.
//   TMEM columns: Q planes 0..63, S -> P planes 64..127, P V 128..191
constexpr int FWD_THREADS = 192;
struct FwdCfg {
  static constexpr int SLOTS = 6;
  static constexpr int SLOT_BYTES = NP * TILE;
  static constexpr int BAR = SLOTS * SLOT_BYTES;
  static constexpr int SMEM = BAR + 256 + 1024;
};

__global__ void __launch_bounds__(FWD_THREADS, 2)
attn_fwd_half_kernel(const float* __restrict__ qmat, const uint8_t* __restrict__ kimg, const uint8_t* __restrict__ vimg,
                   const __grid_constant__ SplitArgs A, float* __restrict__ o, float* __restrict__ lse, uint8_t* __restrict__ pick, uint8_t* __restrict__ fma,
                   AtcDims D, int32_t* __restrict__ dev_err) {
  fb_after_previous();
  using cfg = FwdCfg;
  constexpr int S = cfg::SLOTS;
  enum { B_FULL = 0, B_FREE = S, B_QREADY = 2 * S, B_SFULL, B_PREADY, B_OFULL, B_COUNT };
  extern __shared__ uint8_t smem_raw[];
  const Shared sh = aligned_smem(smem_raw);
  const uint32_t sb = sh.sb, bar0 = sb + cfg::BAR;
  auto bar = [&](int i) { return bar0 + 8u * (uint32_t)i; };
  volatile uint32_t* s_tmem = (volatile uint32_t*)(sh.smem + cfg::BAR + 8 * B_COUNT);
  volatile int* s_abort = (volatile int*)(s_tmem + 1);
  volatile int* s_skip = (volatile int*)(s_tmem + 2);

  const int warp = uniform_warp(), lane = threadIdx.x & 31;
  // causal: the last query tiles have the most key blocks, so they are scheduled first
  const int64_t i0 = (int64_t)(D.causal ? gridDim.x - 1 - blockIdx.x : blockIdx.x) * QT;
  const int h = blockIdx.y;
  const int64_t b = blockIdx.z, bh = b * D.H + h;
  int64_t kv_end = D.Lk;
  if (D.causal && i0 + QT < kv_end) kv_end = i0 + QT;
  const int nkb = (int)((kv_end + KT - 1) / KT);

  if (threadIdx.x == 0) {
    for (int s = 0; s < S; ++s) {
      mbar_init(bar(B_FULL + s), 1);
      mbar_init(bar(B_FREE + s), 1);
    }
    mbar_init(bar(B_QREADY), 4);
    mbar_init(bar(B_SFULL), 1);
    mbar_init(bar(B_PREADY), 4);
    mbar_init(bar(B_OFULL), 1);
    *s_abort = 0;
    *s_skip = (*(volatile int32_t*)dev_err != 0) ? 1 : 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    fence_proxy_async();
  }
  __shared__ HeadState hs;
  const TileNote* notes = A.notes + bh * 3 * D.max_tiles;
  const int state = head_state(hs, notes, D);
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    pick[bh] = state == 1 ? 1 : 0;
    fma[bh] = state == 2 ? 1 : 0;
  }
  if (state == 1) images_of_three(A, bh, (int)blockIdx.x, (int)gridDim.x);
  if (state != 0 || *s_skip != 0) return;
  if (warp == 1) tmem_alloc(s_tmem, 256u);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = __reduce_or_sync(0xffffffffu, *s_tmem);
  constexpr uint32_t T_R = 64, T_O = 128;

  if (warp == 0) {
    // ---------------------------------------------------------------- producer ---
    if (lane == 0) {
      const int64_t base = bh * D.ktiles * (int64_t)SLOT;
      for (int n = 0; n < 2 * nkb; ++n) {
        const int s = n % S;
        if (n >= S && !mbar_wait(bar(B_FREE + s), (uint32_t)(n / S - 1) & 1u, s_abort)) break;
        mbar_arrive_expect_tx(bar(B_FULL + s), (uint32_t)cfg::SLOT_BYTES);
        bulk_load(sb + (uint32_t)(s * cfg::SLOT_BYTES), ((n & 1) ? vimg : kimg) + base + (int64_t)(n >> 1) * SLOT,
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
        mma_rows_t(tmem + T_R, tmem, sb + (uint32_t)(s * cfg::SLOT_BYTES), nks);
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
        mma_planes(tmem + T_O, tmem + T_R, sb + (uint32_t)(s * cfg::SLOT_BYTES), nv);
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
    int sq;
    row_to_tmem(qmat + (b * D.Lq + gi) * D.E + (int64_t)h * D.d, D.d, live, D.vec != 0, t_row, SH_QK, sq);
    tc_wait_st();
    tc_fence_before();
    __syncwarp();
    if (lane == 0) mbar_arrive(bar(B_QREADY));
    auto shift_at = [&](int i) { const int v = __ldg(&notes[i].shift); return v == SH_ZERO ? 0 : v; };   // of the K tiles, then of the V tiles
    int sk_j = shift_at(0), sv_j = shift_at(D.max_tiles);
    float m = -INFINITY, l = 0.0f, fv = 0.0f;         // fv: the scale of the weights and of the V tile whose product is on its way
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
        for (int c = 0; c < 32; ++c) acc[32 * hf + c] = fmaf(__uint_as_float(v[c]), fv, acc[32 * hf + c]);
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
      const float sc = D.scale_log2 * pow2(-(sq + sk_j));
      fv = pow2(-15 - sv_j);
      if (j + 1 < nkb) {
        sk_j = shift_at(j + 1);
        sv_j = shift_at(D.max_tiles + j + 1);
      }
      const float m_new = fmaxf(m, fmaxf(mx0, mx1) * sc);
      const float m_use = (m_new == -INFINITY) ? 0.0f : m_new;
      const float alpha = fast_exp2(m - m_use);   // m = -inf gives 0
      float rs0 = 0.0f, rs1 = 0.0f;
#pragma unroll
      for (int c = 0; c < 32; ++c) {
        const float p = fast_exp2(fmaf(__uint_as_float(s0[c]), sc, -m_use));
        rs0 += p;
        s0[c] = __float_as_uint(p * 32768.0f);
      }
      store_planes32(t_row + T_R, t_row + T_R + 16u, s0);
#pragma unroll
      for (int c = 0; c < 32; ++c) {
        const float p = fast_exp2(fmaf(__uint_as_float(s1[c]), sc, -m_use));
        rs1 += p;
        s1[c] = __float_as_uint(p * 32768.0f);
      }
      store_planes32(t_row + T_R + 32u, t_row + T_R + 48u, s1);
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
        store_row32<false>(o + off, 32 * hf, D.dv, D.vec != 0, acc + 32 * hf, inv);
      }
      lse[bh * D.Lq + gi] = (l > 0.0f) ? fmaf(m, LN2_HI, fmaf(m, LN2_LO, logf(l))) : -INFINITY;
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    __syncwarp();
    tmem_free(tmem, 256u);
  }
  if (threadIdx.x == 0 && *s_abort != 0) atomicExch(dev_err, 4002);
}

// ----------------------------------------------------------------------------------------------------------- dQ ---
// One CTA owns 128 queries of one (batch, head).  Q and dO of those queries live in tensor memory for the whole kernel.
// For every block of 64 keys: S = Q K' and dP = dO V', the compute warps turn them into dS = P (dP - delta) with
// P = exp(S / sqrt(d) - lse) and put its planes over them, and dQ += dS K with the same K tile read MN-major.  Two S / dP
// regions and two sets of four compute warps take the blocks in turn: the tensor cores work on block j + 1 and on dQ of
// block j - 1 while a set is busy with block j.  dQ accumulates in tensor memory over at most 32 blocks (2048 keys: the
// adds truncate), upper products and cross terms apart.
//   TMEM columns: Q planes 0..63, dO planes 64..127, two regions of 128 (S -> dS planes, dP) 128..383, dQ 384..447, cross terms 448..511
//
// Scales.  With s the shifts, scores come times 2^(sq + sk), dP times 2^(sdo + sv).  dS is made in units of 2^-(sdo + svmin): |dP| and
// |delta| are sums of at most 64 products below 2^30, so |dS| < 2^37 there, and 2^-22 of it fits a half; a K tile's shift above the
// least one goes into it too, so that all blocks add up in one scale.
constexpr int SH_SPREAD = 8;   // what the shifts of the K, V, Q and dO tiles of a head may differ by, added up (ordinary ones: by 4)

// The shifts of a head's tiles (those of tiles of zeros, whatever is multiplied with them, are the least ones), their least ones; returns how the
// head is computed.  All threads; ends with a barrier.
struct HeadShifts {
  HeadState head;
  int16_t tile[4][BWD_MAX_BLOCKS];   // K, V, Q, dO: as far as there is room (of the operand that a kernel walks there is)
  int least[4], most[4];
};
__device__ __forceinline__ int head_shifts(HeadShifts& S, const TileNote* notes, const AtcDims& D) {
  if (threadIdx.x < 4) {
    S.least[threadIdx.x] = SH_ZERO;
    S.most[threadIdx.x] = -SH_ZERO;
  }
  if (threadIdx.x == 0) S.head = HeadState{0u, 0u, 0u};
  __syncthreads();
  auto each = [&](auto f) {
    for (int i = threadIdx.x; i < 4 * D.max_tiles; i += (int)blockDim.x) {
      const int job = i / D.max_tiles, t = i - job * D.max_tiles;
      if (t < (job < 2 ? D.ktiles : D.qtiles)) f(job, t, __ldg((const uint2*)(notes + i)));
    }
  };
  each([&](int job, int, uint2 w) {
    S.head.add(job, w);
    const int v = (int16_t)(w.y & 0xffffu);
    if (v == SH_ZERO) return;
    atomicMin(&S.least[job], v);
    atomicMax(&S.most[job], v);
  });
  __syncthreads();
  each([&](int job, int t, uint2 w) {
    const int v = (int16_t)(w.y & 0xffffu);
    if (t < BWD_MAX_BLOCKS) S.tile[job][t] = (int16_t)(v == SH_ZERO ? (S.least[job] == SH_ZERO ? 0 : S.least[job]) : v);
  });
  int spread = 0;
#pragma unroll
  for (int j = 0; j < 4; ++j)
    if (S.most[j] >= S.least[j]) spread += S.most[j] - S.least[j];
  const int state = S.head.state(D);
  __syncthreads();
  return state == 0 && spread > SH_SPREAD ? 1 : state;
}
// the least shift of a job (0 where all tiles are zeros)
__device__ __forceinline__ int least_of(const HeadShifts& S, int job) { return S.least[job] == SH_ZERO ? 0 : S.least[job]; }
struct DqCfg {
  static constexpr int SLOTS = 6;
  static constexpr int SLOT_BYTES = 2 * NP * TILE;   // K tile, V tile
  static constexpr int BAR = SLOTS * SLOT_BYTES;
  static constexpr int SMEM = BAR + 256 + 1024;
};

__global__ void __launch_bounds__(BWD_THREADS, 1)
attn_bwd_dq_half_kernel(const float* __restrict__ q, const float* __restrict__ dout, const uint8_t* __restrict__ kimg,
                      const uint8_t* __restrict__ vimg, const float2* __restrict__ rv, const __grid_constant__ SplitArgs A,
                      uint8_t* __restrict__ pick, uint8_t* __restrict__ fma, int first, float* __restrict__ dq, AtcDims D, int32_t* __restrict__ dev_err) {
  fb_after_previous();
  using cfg = DqCfg;
  constexpr int S = cfg::SLOTS;
  enum { B_FULL = 0, B_FREE = S, B_QREADY = 2 * S, B_SFULL, B_DSREADY = B_SFULL + 2, B_DONE = B_DSREADY + 2, B_COUNT };
  extern __shared__ uint8_t smem_raw[];
  const Shared sh = aligned_smem(smem_raw);
  const uint32_t sb = sh.sb, bar0 = sb + cfg::BAR;
  auto bar = [&](int i) { return bar0 + 8u * (uint32_t)i; };
  volatile uint32_t* s_tmem = (volatile uint32_t*)(sh.smem + cfg::BAR + 8 * B_COUNT);
  volatile int* s_abort = (volatile int*)(s_tmem + 1);
  volatile int* s_skip = (volatile int*)(s_tmem + 2);

  __shared__ HeadShifts hs;
  __shared__ int16_t row_q[QT], row_d[QT];
  const int warp = uniform_warp(), lane = threadIdx.x & 31;
  const int64_t i0 = (int64_t)(D.causal ? gridDim.x - 1 - blockIdx.x : blockIdx.x) * QT;
  const int h = blockIdx.y;
  const int64_t b = blockIdx.z, bh = b * D.H + h;
  int64_t kv_end = D.Lk;
  if (D.causal && i0 + QT < kv_end) kv_end = i0 + QT;
  const int nkb = (int)((kv_end + KT - 1) / KT);

  if (threadIdx.x == 0) {
    for (int s = 0; s < S; ++s) {
      mbar_init(bar(B_FULL + s), 1);
      mbar_init(bar(B_FREE + s), 1);
    }
    mbar_init(bar(B_QREADY), 8);
    for (int r = 0; r < 2; ++r) {
      mbar_init(bar(B_SFULL + r), 1);
      mbar_init(bar(B_DSREADY + r), 4);
    }
    mbar_init(bar(B_DONE), 1);
    *s_abort = 0;
    *s_skip = (*(volatile int32_t*)dev_err != 0) ? 1 : 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    fence_proxy_async();
  }
  const TileNote* notes = A.notes + bh * 4 * D.max_tiles;
  const int state = head_shifts(hs, notes, D);
  if (first) {   // (the dK / dV kernel has not been launched)
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      pick[bh] = state == 1 ? 1 : 0;
      fma[bh] = state == 2 ? 1 : 0;
    }
    if (state == 1) images_of_three(A, bh, (int)blockIdx.x, (int)gridDim.x);
  }
  if (state != 0 || *s_skip != 0) return;
  if (warp == 1) tmem_alloc(s_tmem, 512u);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = __reduce_or_sync(0xffffffffu, *s_tmem);
  constexpr uint32_t T_DO = 64, T_R = 128, T_DQ = 384, T_DX = 448;

  if (warp == 0) {
    // ---------------------------------------------------------------- producer ---
    if (lane == 0) {
      const int64_t base = bh * D.ktiles * (int64_t)SLOT;
      for (int j = 0; j < nkb; ++j) {
        const int s = j % S;
        if (j >= S && !mbar_wait(bar(B_FREE + s), (uint32_t)(j / S - 1) & 1u, s_abort)) break;
        mbar_arrive_expect_tx(bar(B_FULL + s), (uint32_t)cfg::SLOT_BYTES);
        const uint32_t dst = sb + (uint32_t)(s * cfg::SLOT_BYTES);
        const int64_t off = base + (int64_t)j * SLOT;
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
          mma_planes_sum(tmem + T_DQ, tmem + T_DX, r, sb + (uint32_t)((j % S) * cfg::SLOT_BYTES), nd, j > 0);
          tc_commit(bar(B_FREE + j % S));
          if (j == nkb - 1) tc_commit(bar(B_DONE));
        }
        const int t = j + 2, s = t % S;
        if (t < nkb) {
          ok = warp_wait(bar(B_FULL + s), (uint32_t)(t / S) & 1u, s_abort);
          if (!ok) break;
          tc_fence_after();
          const uint32_t base = sb + (uint32_t)(s * cfg::SLOT_BYTES), r = tmem + T_R + (uint32_t)(128 * (t & 1));
          mma_rows_t(r, tmem, base, nks);
          mma_rows_t(r + 64u, tmem + T_DO, base + NP * TILE, nvs);
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
    // the first set brings Q into tensor memory, the second dO
    int sh;
    if (set == 0) row_to_tmem(q + (b * D.Lq + gi) * D.E + (int64_t)h * D.d, D.d, live, D.vec != 0, t_row, SH_QK, sh);
    else row_to_tmem(dout + (b * D.Lq + gi) * D.Ev + (int64_t)h * D.dv, D.dv, live, D.vec != 0, t_row + T_DO, SH_DO, sh);
    (set == 0 ? row_q : row_d)[32 * qd + lane] = (int16_t)sh;
    tc_wait_st();
    tc_fence_before();
    __syncwarp();
    if (lane == 0) mbar_arrive(bar(B_QREADY));
    asm volatile("bar.sync 1, 256;" ::: "memory");   // (compute warps: the rows' shifts)
    const int sq = row_q[32 * qd + lane], sdo = row_d[32 * qd + lane], svmin = least_of(hs, 1), skmin = least_of(hs, 0);
    const float2 ld = rv[bh * ((int64_t)D.qtiles * KT) + gi];   // {inf, 0} past the end: the weights become 0
    const float delta = times_pow2(ld.y, sdo + svmin);
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
      const float sc = D.scale_log2 * pow2(-(sq + hs.tile[0][j])), g = pow2(skmin - hs.tile[0][j] - 22), f = pow2(svmin - hs.tile[1][j]) * g, dg = delta * g;
#pragma unroll
      for (int hf = 0; hf < 2; ++hf) {
        uint32_t sv[32], dp[32];
        tc_ld_32x32b_x32(r + 32u * hf, sv);
        tc_ld_32x32b_x32(r + 64u + 32u * hf, dp);
        tc_wait_ld();
        if (nvalid >= KT) {
#pragma unroll
          for (int c = 0; c < 32; ++c)
            sv[c] = __float_as_uint(fast_exp2(fmaf(__uint_as_float(sv[c]), sc, -ld.x)) * fmaf(__uint_as_float(dp[c]), f, -dg));
        } else {
#pragma unroll
          for (int c = 0; c < 32; ++c) {
            float p = fast_exp2(fmaf(__uint_as_float(sv[c]), sc, -ld.x));
            if (c + 32 * hf >= nvalid) p = 0.0f;
            sv[c] = __float_as_uint(p * fmaf(__uint_as_float(dp[c]), f, -dg));
          }
        }
        store_planes32(r + 32u * hf, r + 32u * hf + 16u, sv);   // (columns this thread has read already)
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
      uint32_t v[32], w[32];
      tc_ld_32x32b_x32(t_row + T_DQ + 32u * set, v);
      tc_ld_32x32b_x32(t_row + T_DX + 32u * set, w);
      tc_wait_ld();
      const int e = 22 - sdo - svmin - skmin;
#pragma unroll
      for (int c = 0; c < 32; ++c) v[c] = __float_as_uint(times_pow2(fmaf(__uint_as_float(w[c]), 0.00048828125f, __uint_as_float(v[c])) * D.scale, e));
      if (live)
        store_row32<false>(dq + (b * D.Lq + gi) * D.E + (int64_t)h * D.d, 32 * set, D.d, D.vec != 0, (const float*)v, 1.0f);
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    __syncwarp();
    tmem_free(tmem, 512u);
  }
  if (threadIdx.x == 0 && *s_abort != 0) atomicExch(dev_err, 4003);
}

// ------------------------------------------------------------------------------------------------------ dK, dV ---
// Transposed, so that keys are the rows (TMEM lanes) of every accumulator.  One CTA owns 128 keys of one (batch, head); K
// and V stay in shared memory as A operands.  For every block of 64 queries:
//   S' = K Q'  and  dP' = V dO'    (B operands: the Q and dO tiles, K-major)
//   P' = exp(S' / sqrt(d) - lse_q),  dS' = P' (dP' - delta_q)     (compute warps; planes back into tensor memory)
//   dV += P' dO  and  dK += dS' Q   (B operands: the same Q and dO tiles, MN-major)
// As in the dQ kernel two regions and two sets of compute warps take the blocks in turn.  The ring of tile slots holds dO0 Q0 dO1 Q1
// dO2 ...; dV is issued before dK and dP' before S', so that a slot freed by dV of block i is reloaded under dK of block i and dP' of
// block i + 2.  K and V in tensor memory would leave room for one region only; from shared memory an MMA of 128 x 64 x 16 takes 48
// clocks, from tensor memory 44.
//   TMEM columns: two regions of 128 (S' -> P' planes, dP' -> dS' planes) 0..255, dV 256..319, its cross terms 320..383, dK and its
//   cross terms 384..511
// Scales as in the dQ kernel: dS' in units of 2^-(sv of the key's tile + sdomin), P' times 2^15; the shifts of the dO and Q tiles above the
// least ones go into P' and dS'.
struct KvCfg {
  // Compute warps per set: eight with half a row of a block each (four, a thread with a whole row: 659 us, here 579 - 618; batch 8, 16 heads, 2048 x
  // 2048, causal).  The dQ kernel gains nothing from it (499 -> 517).
  static constexpr int HALVES = 2;
  static constexpr int THREADS = 64 + 256 * HALVES;
  static constexpr int SLOTS = 8;
  static constexpr int SLOT_BYTES = NP * TILE + 1024;   // a tile and, behind dO, {lse, delta} of its 64 queries
  static constexpr int K_OFF = SLOTS * SLOT_BYTES, V_OFF = K_OFF + NP * 2 * TILE;
  static constexpr int BAR = V_OFF + NP * 2 * TILE;
  static constexpr int SMEM = BAR + 256 + 1024;
};

__global__ void __launch_bounds__(KvCfg::THREADS, 1)
attn_bwd_dkdv_half_kernel(const uint8_t* __restrict__ qimg, const uint8_t* __restrict__ doimg, const uint8_t* __restrict__ kimg,
                        const uint8_t* __restrict__ vimg, const float2* __restrict__ rv, const __grid_constant__ SplitArgs A,
                        uint8_t* __restrict__ pick, uint8_t* __restrict__ fma, float* __restrict__ dk, float* __restrict__ dv, AtcDims D,
                        int32_t* __restrict__ dev_err) {
  fb_after_previous();
  using cfg = KvCfg;
  constexpr int S = cfg::SLOTS;
  enum { B_FULL = 0, B_FREE = S, B_KV = 2 * S, B_SFULL, B_PREADY = B_SFULL + 2, B_DONE = B_PREADY + 2, B_COUNT };
  extern __shared__ uint8_t smem_raw[];
  const Shared sh = aligned_smem(smem_raw);
  const uint32_t sb = sh.sb, bar0 = sb + cfg::BAR;
  auto bar = [&](int i) { return bar0 + 8u * (uint32_t)i; };
  volatile uint32_t* s_tmem = (volatile uint32_t*)(sh.smem + cfg::BAR + 8 * B_COUNT);
  volatile int* s_abort = (volatile int*)(s_tmem + 1);
  volatile int* s_skip = (volatile int*)(s_tmem + 2);

  __shared__ HeadShifts hs;
  const int warp = uniform_warp(), lane = threadIdx.x & 31;
  const int64_t j0 = (int64_t)blockIdx.x * QT;   // first key of this CTA
  const int h = blockIdx.y;
  const int64_t b = blockIdx.z, bh = b * D.H + h;
  // query blocks that see these keys: all of them, or under a causal mask those from the diagonal on
  const int ib0 = D.causal ? (int)(j0 / KT) : 0;
  const int nqb = (int)((D.Lq + KT - 1) / KT) - ib0;   // may be <= 0: nothing attends to these keys

  if (threadIdx.x == 0) {
    for (int s = 0; s < S; ++s) {
      mbar_init(bar(B_FULL + s), 1);
      mbar_init(bar(B_FREE + s), 1);
    }
    mbar_init(bar(B_KV), 1);
    for (int r = 0; r < 2; ++r) {
      mbar_init(bar(B_SFULL + r), 1);
      mbar_init(bar(B_PREADY + r), 4 * cfg::HALVES);
    }
    mbar_init(bar(B_DONE), 1);
    *s_abort = 0;
    *s_skip = (*(volatile int32_t*)dev_err != 0) ? 1 : 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    fence_proxy_async();
  }
  const TileNote* notes = A.notes + bh * 4 * D.max_tiles;
  const int state = head_shifts(hs, notes, D);
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    pick[bh] = state == 1 ? 1 : 0;
    fma[bh] = state == 2 ? 1 : 0;
  }
  if (state == 1) images_of_three(A, bh, (int)blockIdx.x, (int)gridDim.x);
  if (state != 0 || *s_skip != 0) return;
  if (warp == 1) tmem_alloc(s_tmem, 512u);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = __reduce_or_sync(0xffffffffu, *s_tmem);
  constexpr uint32_t T_DV = 256, T_DK = 384;   // (their cross terms 64 columns behind)

  if (warp == 0) {
    // ---------------------------------------------------------------- producer ---
    if (lane == 0 && nqb > 0) {
      mbar_arrive_expect_tx(bar(B_KV), (uint32_t)(4 * NP * TILE));
#pragma unroll
      for (int p = 0; p < NP; ++p)
#pragma unroll
        for (int t = 0; t < 2; ++t) {   // plane p of the CTA's two 64-key tiles, one after the other
          const int64_t off = (bh * D.ktiles + 2 * (int64_t)blockIdx.x + t) * SLOT + p * TILE;
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
        bulk_load(dst, (is_do ? doimg : qimg) + tile * (int64_t)SLOT, NP * TILE, bar(B_FULL + s));
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
          const uint32_t r = tmem + (uint32_t)(128 * (i & 1));
          mma_planes_sum(tmem + T_DV, tmem + T_DV + 64u, r, slot(2 * i), nv, i > 0);
          tc_commit(bar(B_FREE + (2 * i) % S));
          mma_planes_sum(tmem + T_DK, tmem + T_DK + 64u, r + 64u, slot(2 * i + 1), nd, i > 0);
          tc_commit(bar(B_FREE + (2 * i + 1) % S));
          if (i == nqb - 1) tc_commit(bar(B_DONE));
        }
        const int t = i + 2;
        if (t < nqb) {
          const uint32_t r = tmem + (uint32_t)(128 * (t & 1));
          ok = full(2 * t);
          if (!ok) break;
          tc_fence_after();
          mma_rows_s(r + 64u, sb + cfg::V_OFF, slot(2 * t));
          ok = full(2 * t + 1);
          if (!ok) break;
          tc_fence_after();
          mma_rows_s(r, sb + cfg::K_OFF, slot(2 * t + 1));
          tc_commit(bar(B_SFULL + (t & 1)));
        }
      }
    }
  } else {
    // ------------------------------------------------------------ compute warps ---
    constexpr int HV = cfg::HALVES;
    const int set = (warp - 2) / (4 * HV), half = ((warp - 2) >> 2) % HV, qd = warp & 3;
    const int64_t kj = j0 + 32 * qd + lane;   // this thread's key
    const bool live = kj < D.Lk;
    const uint32_t t_row = tmem + ((uint32_t)(32 * qd) << 16);
    auto own_shift = [&](int job) {   // (of the two key tiles of this CTA; there may be more than BWD_MAX_BLOCKS)
      const int v = __ldg(&notes[job * D.max_tiles + 2 * (int64_t)blockIdx.x + (qd >> 1)].shift);
      return v == SH_ZERO ? least_of(hs, job) : v;
    };
    const int skr = own_shift(0), svr = own_shift(1);
    const int sqmin = least_of(hs, 2), sdmin = least_of(hs, 3);
    const float to_units = pow2(svr + sdmin);
    bool ok = true;
    for (int i = set; i < nqb && ok; i += 2) {
      const int n = 2 * i;
      ok = mbar_wait(bar(B_FULL + n % S), (uint32_t)(n / S) & 1u, s_abort) && mbar_wait(bar(B_SFULL + set), (uint32_t)(i >> 1) & 1u, s_abort);
      if (!ok) break;
      tc_fence_after();
      const float4* row = (const float4*)(sh.smem + (n % S) * cfg::SLOT_BYTES + NP * TILE);   // {lse, delta} of two queries
      // queries of the block this key is seen by: query < Lq (dead ones carry lse = inf), and query >= key when causal
      const int64_t i0b = (int64_t)(ib0 + i) * KT;
      int clo = 0;
      if (D.causal && kj - i0b > 0) clo = (kj - i0b) > KT ? KT : (int)(kj - i0b);
      if (!live) clo = KT;
      const uint32_t r = t_row + (uint32_t)(128 * set);
      const int sqi = hs.tile[2][ib0 + i], sdi = hs.tile[3][ib0 + i];
      const float sc = D.scale_log2 * pow2(-(skr + sqi)), pv = pow2(15 + sdmin - sdi), g = pow2(sqmin - sqi - 22), f = pow2(sdmin - sdi) * g,
                  dg = to_units * g;
#pragma unroll
      for (int it = 0; it < 2 / HV; ++it) {
        const int hf = HV == 2 ? half : it;
        uint32_t sv[32], dp[32];
        tc_ld_32x32b_x32(r + 32u * hf, sv);
        tc_ld_32x32b_x32(r + 64u + 32u * hf, dp);
        tc_wait_ld();
#pragma unroll
        for (int c = 0; c < 32; c += 2) {
          const float4 w = row[16 * hf + (c >> 1)];
          float p0 = fast_exp2(fmaf(__uint_as_float(sv[c]), sc, -w.x));
          float p1 = fast_exp2(fmaf(__uint_as_float(sv[c + 1]), sc, -w.z));
          if (c + 32 * hf < clo) p0 = 0.0f;
          if (c + 1 + 32 * hf < clo) p1 = 0.0f;
          sv[c] = __float_as_uint(p0 * pv);
          sv[c + 1] = __float_as_uint(p1 * pv);
          dp[c] = __float_as_uint(p0 * fmaf(__uint_as_float(dp[c]), f, -w.y * dg));
          dp[c + 1] = __float_as_uint(p1 * fmaf(__uint_as_float(dp[c + 1]), f, -w.w * dg));
        }
        // (over columns this thread has read already)
        store_planes32(r + 32u * hf, r + 32u * hf + 16u, sv);
        store_planes32(r + 64u + 32u * hf, r + 80u + 32u * hf, dp);
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
      float* drow = set == 0 ? dv + (b * D.Lk + kj) * D.Ev + (int64_t)h * D.dv : dk + (b * D.Lk + kj) * D.E + (int64_t)h * D.d;
#pragma unroll
      for (int it = 0; it < 2 / HV; ++it) {
        const int hf = HV == 2 ? half : it;
        uint32_t v[32], w[32];
        if (nqb > 0) {
          tc_ld_32x32b_x32(t_row + (set == 0 ? T_DV : T_DK) + 32u * hf, v);
          tc_ld_32x32b_x32(t_row + (set == 0 ? T_DV : T_DK) + 64u + 32u * hf, w);
          tc_wait_ld();
          const int e = set == 0 ? -15 - sdmin : 22 - svr - sdmin - sqmin;
#pragma unroll
          for (int c = 0; c < 32; ++c)
            v[c] = __float_as_uint(times_pow2(fmaf(__uint_as_float(w[c]), 0.00048828125f, __uint_as_float(v[c])) * (set == 0 ? 1.0f : D.scale), e));
        } else {
#pragma unroll
          for (int c = 0; c < 32; ++c) v[c] = 0u;
        }
        if (live) store_row32<false>(drow, 32 * hf, set == 0 ? D.dv : D.d, D.vec != 0, (const float*)v, 1.0f);
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    __syncwarp();
    tmem_free(tmem, 512u);
  }
  if (threadIdx.x == 0 && *s_abort != 0) atomicExch(dev_err, 4004);
}

// Behind the kernels here: the picked heads (attention_tc.cu) and those with values that are not finite (attention.cu).  Launches that find none cost
// 3 - 6 us each.  Batch 8, 16 heads of 64, 2048 x 2048, causal, forward and backward in us: no head picked 420 and 1233, one 505 and 1340, all 630 and
// 2190 (all heads on three bf16 planes from the start: 560 and 2079; one head on the FMA kernels: 2455 and 9377).
int32_t fwd_impl(fb_ctx* ctx, cudaStream_t stream, const float* q, const float* k, const float* v, float* o, float* lse, const AtcPlan& P,
                 int64_t batch) {
  const AtcDims& D = P.D;
  const int64_t note_bytes = (int64_t)D.H * 3 * D.max_tiles * (int64_t)sizeof(TileNote), per = 2 * P.kbytes + note_bytes + 2 * D.H;
  int64_t chunk = IMAGE_BYTES / per;
  chunk = chunk < 1 ? 1 : (chunk > batch ? batch : chunk);
  const fb_temp images(ctx, stream, (size_t)(chunk * per));
  uint8_t* img = (uint8_t*)images.p;
  if (!img) return FB_ERR_UNSUPPORTED;
  FB_ONCE(ctx, FB_CUDA(cudaFuncSetAttribute(attn_fwd_half_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, FwdCfg::SMEM)));
  for (int64_t b0 = 0; b0 < batch; b0 += chunk) {
    const int64_t nb = b0 + chunk > batch ? batch - b0 : chunk;
    const float *qb = q + b0 * D.Lq * D.E, *kb = k + b0 * D.Lk * D.E, *vb = v + b0 * D.Lk * D.Ev;
    float *ob = o + b0 * D.Lq * D.Ev, *lb = lse + b0 * D.H * D.Lq;
    TileNote* notes = (TileNote*)(img + nb * 2 * P.kbytes);
    uint8_t *pick = (uint8_t*)notes + nb * note_bytes, *fma = pick + nb * D.H;   // a byte per head each
    SplitArgs A = {};
    A.H = D.H; A.vec = D.vec; A.notes = notes; A.jobs = 3; A.max_tiles = D.max_tiles;
    A.job[0] = {kb, img, D.Lk, D.E, D.d, D.ktiles, SH_QK};
    A.job[1] = {vb, img + nb * P.kbytes, D.Lk, D.Ev, D.dv, D.ktiles, SH_V};
    A.job[2] = {qb, nullptr, D.Lq, D.E, D.d, D.qtiles, SH_QK};
    fb_launch(attn_half_split_kernel, dim3((unsigned)D.max_tiles, (unsigned)(nb * D.H), 3), SPLIT_THREADS, 0, stream, A);
    FB_LAUNCH_CHECK();
    fb_launch(attn_fwd_half_kernel, dim3((unsigned)(D.qtiles / 2), (unsigned)D.H, (unsigned)nb), FWD_THREADS, FwdCfg::SMEM, stream, qb, img, img + nb * P.kbytes, A, ob, lb,
              pick, fma, D, ctx->dev_error);
    FB_LAUNCH_CHECK();
    int32_t st = fwd_picked(ctx, stream, qb, img, img + nb * P.kbytes, ob, lb, D, nb, pick);
    if (st == FB_OK) st = fb_attn_fwd_redo(ctx, stream, 0, qb, kb, vb, ob, nullptr, lb, D.E, D.Ev, D.Lq, D.Lk, nb, D.H, D.causal, fma, 1);
    if (st != FB_OK) return st;
  }
  return FB_OK;
}

int32_t bwd_impl(fb_ctx* ctx, cudaStream_t stream, const float* q, const float* k, const float* v, const float* o, const float* lse, const float* dout, float* dq,
                 float* dk, float* dv, const AtcPlan& P, int64_t batch, bool do_kv, bool do_q) {
  const AtcDims& D = P.D;
  const int64_t note_bytes = (int64_t)D.H * 4 * D.max_tiles * (int64_t)sizeof(TileNote), per = 2 * P.kbytes + 2 * P.qbytes + P.rvbytes + note_bytes + 2 * D.H;
  int64_t chunk = IMAGE_BYTES / per;
  chunk = chunk < 1 ? 1 : (chunk > batch ? batch : chunk);
  const fb_temp images(ctx, stream, (size_t)(chunk * per));
  uint8_t* img = (uint8_t*)images.p;
  if (!img) return FB_ERR_UNSUPPORTED;
  FB_ONCE(ctx, FB_CUDA(cudaFuncSetAttribute(attn_bwd_dkdv_half_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, KvCfg::SMEM)));
  FB_ONCE(ctx, FB_CUDA(cudaFuncSetAttribute(attn_bwd_dq_half_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, DqCfg::SMEM)));
  for (int64_t b0 = 0; b0 < batch; b0 += chunk) {
    const int64_t nb = b0 + chunk > batch ? batch - b0 : chunk;
    uint8_t *ki = img, *vi = ki + nb * P.kbytes, *qi = vi + nb * P.kbytes, *doi = qi + nb * P.qbytes;
    float2* rv = (float2*)(doi + nb * P.qbytes);
    TileNote* notes = (TileNote*)((uint8_t*)rv + nb * P.rvbytes);
    uint8_t *pick = (uint8_t*)notes + nb * note_bytes, *fma = pick + nb * D.H;
    const int64_t qoff = b0 * D.Lq * D.E, qvoff = b0 * D.Lq * D.Ev, koff = b0 * D.Lk * D.E, kvoff = b0 * D.Lk * D.Ev;
    const float *qb = q + qoff, *kb = k + koff, *vb = v + kvoff, *dob = dout + qvoff, *lb = lse + b0 * D.H * D.Lq;
    float *dqb = do_q ? dq + qoff : nullptr, *dkb = do_kv ? dk + koff : nullptr, *dvb = do_kv ? dv + kvoff : nullptr;
    SplitArgs A = {};
    A.H = D.H; A.vec = D.vec; A.notes = notes; A.jobs = 4; A.max_tiles = D.max_tiles;
    A.job[0] = {kb, ki, D.Lk, D.E, D.d, D.ktiles, SH_QK};
    A.job[1] = {vb, vi, D.Lk, D.Ev, D.dv, D.ktiles, SH_V};
    A.job[2] = {qb, qi, D.Lq, D.E, D.d, D.qtiles, SH_QK};
    A.job[3] = {dob, doi, D.Lq, D.Ev, D.dv, D.qtiles, SH_DO};
    A.o = o + qvoff; A.lse = lb; A.rv = rv;
    fb_launch(attn_half_split_kernel, dim3((unsigned)D.max_tiles, (unsigned)(nb * D.H), 4), SPLIT_THREADS, 0, stream, A);
    FB_LAUNCH_CHECK();
    if (do_kv) {
      fb_launch(attn_bwd_dkdv_half_kernel, dim3((unsigned)(D.ktiles / 2), (unsigned)D.H, (unsigned)nb), KvCfg::THREADS, KvCfg::SMEM, stream, qi, doi, ki, vi, rv, A, pick, fma,
                dkb, dvb, D, ctx->dev_error);
      FB_LAUNCH_CHECK();
    }
    if (do_q) {
      fb_launch(attn_bwd_dq_half_kernel, dim3((unsigned)(D.qtiles / 2), (unsigned)D.H, (unsigned)nb), BWD_THREADS, DqCfg::SMEM, stream, qb, dob, ki, vi, rv, A, pick, fma,
                do_kv ? 0 : 1, dqb, D, ctx->dev_error);
      FB_LAUNCH_CHECK();
    }
    int32_t st = bwd_picked(ctx, stream, qb, dob, ki, vi, qi, doi, rv, dqb, dkb, dvb, D, nb, pick);
    if (st == FB_OK)
      st = fb_attn_bwd_redo(ctx, stream, 0, qb, kb, vb, lb, (const float*)rv + 1, (int64_t)D.qtiles * KT, dob, dqb, dkb, dvb, D.E, D.Ev, D.Lq, D.Lk, nb, D.H, D.causal, fma, 1);
    if (st != FB_OK) return st;
  }
  return FB_OK;
}

}  // namespace

// Both return FB_ERR_UNSUPPORTED when the call is not one these kernels take (the caller then uses the FMA kernels).
int32_t fb_attn_fwd_tc(fb_ctx* ctx, cudaStream_t stream, const float* q, const float* k, const float* v, const uint8_t* mask,
                       float* o, float* lse, int64_t e_dim, int64_t ev_dim, int64_t lq, int64_t lk, int64_t batch, int nheads,
                       int causal) {
  AtcPlan P;
  if (!attn_tc_enabled() || mask != nullptr || !make_plan(&P, 3, e_dim, ev_dim, lq, lk, batch, nheads, causal)) return FB_ERR_UNSUPPORTED;
  if (!fb_aligned16(q) || !fb_aligned16(k) || !fb_aligned16(v) || !fb_aligned16(o)) P.D.vec = 0;
  return fwd_impl(ctx, stream, q, k, v, o, lse, P, batch);
}

// *did_kv, *did_q: which part was done.  dQ, dK and dV accumulate in tensor memory with truncating adds; beyond 2048 keys
// (queries), for the other head sizes and for unaligned arrays, the FMA kernels are the more accurate ones (8 heads of 64,
// 512 x 512: dQ 4e-7, dK and dV 6e-7 of the norm in 245 us, here 1.4e-6 and 5e-6 in 87).
int32_t fb_attn_bwd_tc(fb_ctx* ctx, cudaStream_t stream, const float* q, const float* k, const float* v, const uint8_t* mask, const float* o,
                       const float* lse, const float* dout, float* dq, float* dk, float* dv, int64_t e_dim, int64_t ev_dim, int64_t lq,
                       int64_t lk, int64_t batch, int nheads, int causal, bool* did_kv, bool* did_q) {
  AtcPlan P;
  *did_kv = *did_q = false;
  if (!attn_tc_enabled() || !attn_bwd_tc_enabled() || mask != nullptr || !make_plan(&P, 3, e_dim, ev_dim, lq, lk, batch, nheads, causal) ||
      P.D.d != HD || P.D.dv != HD)
    return FB_ERR_UNSUPPORTED;
  // (arrays off the 16-byte boundary have always been the FMA kernels')
  if (!fb_aligned16(q) || !fb_aligned16(k) || !fb_aligned16(v) || !fb_aligned16(dout)) return FB_ERR_UNSUPPORTED;
  const bool kv = lq <= BWD_MAX_BLOCKS * KT && fb_aligned16(dk) && fb_aligned16(dv), qq = lk <= BWD_MAX_BLOCKS * KT && fb_aligned16(dq);
  if (!kv && !qq) return FB_ERR_UNSUPPORTED;
  if (!fb_aligned16(o)) P.D.vec = 0;
  const int32_t st = bwd_impl(ctx, stream, q, k, v, o, lse, dout, dq, dk, dv, P, batch, kv, qq);
  if (st == FB_OK) {
    *did_kv = kv;
    *did_q = qq;
  }
  return st;
}
