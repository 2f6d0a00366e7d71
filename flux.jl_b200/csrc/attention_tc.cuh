// What the tensor-core attention kernels on bf16 planes (attention_tc.cu) and on half-precision planes (attention_half.cu) share: sizes, instruction
// wrappers, rows in and out of registers, the plan of a call.
#pragma once
#include <cuda.h>
#include <cuda_bf16.h>
#include <stdlib.h>

#include "common.cuh"
#include "tc_common.cuh"

namespace fb_atc {

constexpr int QT = 128;        // rows (queries, or keys in the dK / dV kernel) per CTA
constexpr int KT = 64;         // keys (queries) per block
constexpr int HD = 64;         // padded head size
constexpr int TILE = 8192;     // one plane of a 64 x 64 tile: 64 rows of 128 bytes, 128-byte swizzle
constexpr uint32_t LAYOUT_SW128 = 2;
constexpr float LOG2E = 1.4426950408889634f, LN2_HI = 0.693145751953125f, LN2_LO = 1.42860682030941723e-6f;

struct AtcDims {
  int64_t E, Ev, Lq, Lk;
  int H, causal, d, dv;
  int qtiles, ktiles;   // 64-row tiles per (batch, head) in the plane images (even)
  int max_tiles;        // the larger of both
  int vec;              // rows can be read and written 16 bytes at a time
  float scale_log2;     // log2(e) / sqrt(d)
  float scale;          // 1 / sqrt(d)
};

// --------------------------------------------------------------------------------------------------- wrappers ---
__device__ __forceinline__ void tc_st_32x32b_x16(uint32_t taddr, const uint32_t* r) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
      "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}
__device__ __forceinline__ void tc_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// Shared-memory descriptors travel as their low word (start address / 16 in its 14 low bits, leading offset above), to which a
// step's offset is added, and a high word that all steps share.  A tile ends below 228 KB, so that the sum never leaves the
// 14 bits.  (As 64-bit sums for A and B under a run-time step count one form of the product below gave wrong low-order terms;
// where the compiler went wrong there is not known, so no form adds to 64 bits.)
//
// D[tmem] (+)= A[tmem] * B[smem]: the A tile (128 rows x 16 halves) sits in 8 consecutive TMEM columns, two values each
__device__ __forceinline__ void tc_mma_ta(uint32_t d_tmem, uint32_t a_tmem, uint32_t b_lo, uint32_t hi, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t.reg .b64 db;\n\t"
      "elect.sync _|q, 0xffffffff;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "mov.b64 db, {%2, %9};\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], db, %3, {%5, %6, %7, %8}, p;\n\t}"
      ::"r"(d_tmem), "r"(a_tmem), "r"(b_lo), "r"(idesc), "r"(accumulate), "r"(0u), "r"(0u), "r"(0u), "r"(0u), "r"(hi)
      : "memory");
}
// the same with A from shared memory
__device__ __forceinline__ void tc_mma_sa(uint32_t d_tmem, uint32_t a_lo, uint32_t b_lo, uint32_t hi, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t.reg .b64 da, db;\n\t"
      "elect.sync _|q, 0xffffffff;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "mov.b64 da, {%1, %9};\n\t"
      "mov.b64 db, {%2, %9};\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %3, {%5, %6, %7, %8}, p;\n\t}"
      ::"r"(d_tmem), "r"(a_lo), "r"(b_lo), "r"(idesc), "r"(accumulate), "r"(0u), "r"(0u), "r"(0u), "r"(0u), "r"(hi)
      : "memory");
}

// plain bulk copy of a piece of a plane image (both addresses and the size are multiples of 16 bytes)
__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(dst), "l"(src), "r"(bytes), "r"(bar)
               : "memory");
}

// 2^x by the special-function unit (relative error ~2^-22, far inside the tolerance of a softmax weight)
__device__ __forceinline__ float fast_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

__device__ __forceinline__ uint32_t pack2(float lo, float hi) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&v);
}

// Two values as three bf16 planes (x in the low half of each word): truncation to the upper 16 bits leaves a remainder of
// at most 16 significant bits, the same again one of at most 8, which is a bf16 value.
__device__ __forceinline__ void split3(float x, float y, uint32_t& p0, uint32_t& p1, uint32_t& p2) {
  const uint32_t xb = __float_as_uint(x), yb = __float_as_uint(y);
  p0 = __byte_perm(xb, yb, 0x7632);
  const float rx = x - __uint_as_float(xb & 0xffff0000u), ry = y - __uint_as_float(yb & 0xffff0000u);
  const uint32_t rxb = __float_as_uint(rx), ryb = __float_as_uint(ry);
  p1 = __byte_perm(rxb, ryb, 0x7632);
  p2 = __byte_perm(__float_as_uint(rx - __uint_as_float(rxb & 0xffff0000u)), __float_as_uint(ry - __uint_as_float(ryb & 0xffff0000u)), 0x7632);
}
// 32 consecutive features (from c0) of one row as Float32 values; zero beyond the head size or for a dead row
__device__ __forceinline__ void row_f32(const float* src, int c0, int width, bool live, bool vec, uint32_t* v) {
  if (vec) {
#pragma unroll
    for (int c = 0; c < 32; c += 4) {
      float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
      if (live && c0 + c < width) x = __ldg((const float4*)(src + c0 + c));
      v[c] = __float_as_uint(x.x); v[c + 1] = __float_as_uint(x.y); v[c + 2] = __float_as_uint(x.z); v[c + 3] = __float_as_uint(x.w);
    }
  } else {
#pragma unroll
    for (int c = 0; c < 32; ++c) v[c] = (live && c0 + c < width) ? __float_as_uint(__ldg(src + c0 + c)) : 0u;
  }
}

__device__ __forceinline__ bool not_finite(uint32_t bits) { return (bits & 0x7f800000u) == 0x7f800000u; }

// 32 columns (from c0) of an output row, scaled; Float32, or bf16 rounded to nearest
template <bool BF16>
__device__ __forceinline__ void store_row32(void* dst, int c0, int width, bool vec, const float* v, float sc) {
  if (BF16) {
#pragma unroll
    for (int c = 0; c < 32; c += 8)
      if (c0 + c < width)
        *(uint4*)((uint16_t*)dst + c0 + c) = make_uint4(pack2(v[c] * sc, v[c + 1] * sc), pack2(v[c + 2] * sc, v[c + 3] * sc),
                                                        pack2(v[c + 4] * sc, v[c + 5] * sc), pack2(v[c + 6] * sc, v[c + 7] * sc));
  } else if (vec) {
#pragma unroll
    for (int c = 0; c < 32; c += 4)
      if (c0 + c < width) *(float4*)((float*)dst + c0 + c) = make_float4(v[c] * sc, v[c + 1] * sc, v[c + 2] * sc, v[c + 3] * sc);
  } else {
#pragma unroll
    for (int c = 0; c < 32; ++c)
      if (c0 + c < width) ((float*)dst)[c0 + c] = v[c] * sc;
  }
}

// operand tiles at 1024-byte boundaries: K-major (one k-step of 16 values = 32 bytes) and MN-major (16 rows of 128 bytes)
__device__ __forceinline__ uint64_t desc_k(uint32_t saddr) { return make_smem_desc(saddr, 16, 1024, LAYOUT_SW128); }
__device__ __forceinline__ uint64_t desc_mn(uint32_t saddr) { return make_smem_desc(saddr, KT * 128, 1024, LAYOUT_SW128); }

// ---------------------------------------------------------------------------------- what the kernels share ---
struct Shared {
  uint8_t* smem;
  uint32_t sb;       // its shared-space address (1024-byte aligned)
};
__device__ __forceinline__ Shared aligned_smem(uint8_t* raw) {
  Shared s;
  s.smem = (uint8_t*)(((uintptr_t)raw + 1023) & ~(uintptr_t)1023);
  s.sb = smem_u32(s.smem);
  return s;
}
__device__ __forceinline__ void tmem_alloc(volatile uint32_t* slot, uint32_t cols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32((const void*)slot)), "r"(cols) : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_free(uint32_t base, uint32_t cols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(base), "r"(cols) : "memory");
}

constexpr int BWD_THREADS = 320;
constexpr int BWD_MAX_BLOCKS = 32;   // blocks whose products the backward kernels add up in tensor memory at most (the adds truncate)

// ------------------------------------------------------------------------------------------------------- host side ---
// FLUXB200_ATTN_TC = 0 keeps attention on the Float32 FMA kernels, FLUXB200_ATTN_BWD_TC = 0 its backward pass.
inline bool env_on(const char* name) {
  const char* e = getenv(name);
  return !(e != nullptr && e[0] == '0');
}
inline bool attn_tc_enabled() {
  static const bool on = env_on("FLUXB200_ATTN_TC");
  return on;
}
inline bool attn_bwd_tc_enabled() {
  static const bool on = env_on("FLUXB200_ATTN_BWD_TC");
  return on;
}

// the plane images of one call take at most this much memory unless one batch entry needs more: a call is cut along the batch
// otherwise
constexpr int64_t IMAGE_BYTES = (int64_t)512 << 20;

struct AtcPlan {
  AtcDims D;
  int64_t qbytes, kbytes;   // image of one batch entry's Q (dO), K (V)
  int64_t rvbytes;
};

inline bool make_plan(AtcPlan* P, int np, int64_t e_dim, int64_t ev_dim, int64_t lq, int64_t lk, int64_t batch, int nheads, int causal) {
  if (nheads < 1 || lq < 1 || lk < 1 || batch < 1 || batch > 65535 || nheads > 65535) return false;
  const int64_t d = e_dim / nheads, dv = ev_dim / nheads;
  if (d < 1 || dv < 1 || d > HD || dv > HD) return false;
  if (np == 1 && (d % 8 != 0 || dv % 8 != 0)) return false;
  if (lq > 0x3fffff00 || lk > 0x3fffff00) return false;
  AtcDims& D = P->D;
  D.E = e_dim; D.Ev = ev_dim; D.Lq = lq; D.Lk = lk; D.H = nheads; D.causal = causal ? 1 : 0;
  D.d = (int)d; D.dv = (int)dv;
  D.qtiles = (int)((lq + QT - 1) / QT) * 2;
  D.ktiles = (int)((lk + QT - 1) / QT) * 2;
  D.max_tiles = D.qtiles > D.ktiles ? D.qtiles : D.ktiles;
  D.vec = (d % 4 == 0 && dv % 4 == 0) ? 1 : 0;   // with 16-byte aligned arrays every row of a head is 16-byte aligned
  D.scale = 1.0f / sqrtf((float)d);
  D.scale_log2 = D.scale * LOG2E;
  P->qbytes = (int64_t)nheads * D.qtiles * np * TILE;
  P->kbytes = (int64_t)nheads * D.ktiles * np * TILE;
  P->rvbytes = (int64_t)nheads * D.qtiles * KT * (int64_t)sizeof(float2);
  return true;
}

// attention_tc.cu: Float32 heads on three bf16 planes, those with a byte of `pick` set (one per (batch, head)).  Images of three planes a tile;
// dq, or dk and dv, may be NULL.
int32_t fwd_picked(fb_ctx* ctx, cudaStream_t stream, const float* q, const uint8_t* kimg, const uint8_t* vimg, float* o, float* lse, const AtcDims& D, int64_t batch,
                   const uint8_t* pick);
int32_t bwd_picked(fb_ctx* ctx, cudaStream_t stream, const float* q, const float* dout, const uint8_t* kimg, const uint8_t* vimg, const uint8_t* qimg,
                   const uint8_t* doimg, const float2* rv, float* dq, float* dk, float* dv, const AtcDims& D, int64_t batch, const uint8_t* pick);

}  // namespace fb_atc
