// Float32 operands of a product as images of two half-precision planes, which the tensor cores multiply at twice the TF32 rate
// (gemm_tc.cu).
//
// x 2^s = hi + lo + r, hi and lo rounded to nearest: 11 + 11 bits and two signs, |r| <= 2^-23 |x 2^s| as long as lo is a normal
// number.  Half precision has 5 bits of exponent, so every row (the k-values that meet in one sum) has a power of two s of its own
// that puts its largest magnitude into [2^15, 2^16); the product's epilogue takes it back, exactly.  |r| <= 2^-25 for an element whose
// lo is not normal, which is 2^-19 of it from 1/64 of the scaled row on (2^-21 to 2^-22 of the row's largest) and 2^-17 from 1/256 on.
// Smaller elements may be all that an element of the product is made of (the other operand's row may be zero, or small, where
// this one is large), so the images leave them out: they are listed row by row and the product's epilogue adds them in Float32.
// The line lies where the error against sum |a||b| over an element's own terms stays below that of 3xTF32, which is off by 7.3e-9 for
// each of min(K, 2048) k-values: 1/256 from K = 2048 on (2^-17 + 1.8e-6 against 1.5e-5), else 1/64 (2^-19 + 1.8e-6 against 7.5e-6 at 1024).
// Of 4096 N(0, 1) values 0.001 are left out, of the gradients behind a gelu 0.03; with the line at 1/12 it was 0.024 and 0.4, and the
// products of a training step of 4096 x 4096 layers took 1.4 times as long, with 1/64 1.15 times.
// A row with more of them than its list holds sets a word that turns the product to 3xTF32.
// A row that holds an infinity or a NaN gives NaN, as in 3xTF32.
//
// Image: 128 rows x 64 k-values, plane hi then plane lo, each as the 128-byte rows that one TMA box of 256 rows brings into
// shared memory in the 128-byte swizzle: [128][64 k] for a K-major operand, [2][64 k][64 rows] for an MN-major one.  So the
// product needs one load per operand and stage whatever the operand's order, no transposition and no bounds.  k-values beyond K
// are zero; rows beyond the operand's hold anything (their sums are not stored).
//
// Bound: HBM.  A K-major operand is read once (a row stays in registers up to 8192 k-values) and written once, 8 bytes an
// element; an MN-major one is read once more for its rows' largest values (partial maxima of up to 16 ranges of k, which the
// second kernel puts together), from L2 where it fits.
#include <cuda_fp16.h>

#include "common.cuh"

namespace {

constexpr int IMG_ROWS = 128, IMG_K = 64, IMG_HALVES = IMG_ROWS * IMG_K;   // halves of one plane of an image
constexpr int MAX_CHUNKS = 16;

struct PlaneOp {
  const float* src;
  int64_t ld;
  int rows, K, num_kb, mn_major;
  uint16_t* img;
  int32_t* exps;       // [rows, padded to 128]: the exponent that undoes a row's scale
  uint32_t* part;      // MN-major: [chunks][rows, padded to 128] partial maxima
  int32_t* left;       // elements of a row that its image leaves out, and where they are listed
  int2* list;
  int cap;
  int32_t* over;
  float least;         // the scaled magnitude from which on the images hold an element
  int chunks, chunk_k;
  int blocks1, blocks2;   // blocks of the first and second kernel
};

// power of two that puts a row's largest magnitude (given as its bits) into [2^15, 65504], or just below 2^15 where that would be above
__device__ __forceinline__ int row_shift(uint32_t max_bits) {
  const int e = (int)(max_bits >> 23);
  const int s = ((max_bits & 0x7fffffu) > 0x7fe000u ? 141 : 142) - e;
  return max_bits == 0 ? 0 : s > 126 ? 126 : s < -112 ? -112 : s;
}
__device__ __forceinline__ uint32_t abs_bits(float x) { return __float_as_uint(x) & 0x7fffffffu; }

// element k of a row goes on the row's list, scaled.  (One below 2^-50 leaves the product to 3xTF32: here its products could underflow.)
__device__ __noinline__ void list_element(int32_t* left, int2* list, int cap, int32_t* over, int row, int k, float x) {
  const int i = atomicAdd(left + row, 1);
  if (i < cap && fabsf(x) >= 0x1p-50f) list[(int64_t)row * cap + i] = make_int2(k, (int)__float_as_uint(x));
  else *(volatile int32_t*)over = 1;
}
// element (row0 + j drow, k0 + j dk) = x[j]: those that the images leave out go on the lists and become zero
__device__ __forceinline__ void leave_out8(const PlaneOp& op, float (&x)[8], const float (&sc)[8], int row0, int drow, int k0, int dk) {
  bool any = false;
#pragma unroll
  for (int j = 0; j < 8; ++j) any |= fb_planes_leaves_out(x[j], sc[j], op.least);
  if (!any) return;
#pragma unroll
  for (int j = 0; j < 8; ++j)
    if (fb_planes_leaves_out(x[j], sc[j], op.least)) {
      list_element(op.left, op.list, op.cap, op.over, row0 + j * drow, k0 + j * dk, x[j] * sc[j]);
      x[j] = 0.0f;
    }
}

// 8 values -> 8 upper and 8 lower halves
__device__ __forceinline__ void split8(const float (&x)[8], const float (&sc)[8], uint4& hi, uint4& lo) {
  uint32_t h[4], l[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float a = x[2 * i] * sc[2 * i], b = x[2 * i + 1] * sc[2 * i + 1];
    const __half2 h2 = __floats2half2_rn(a, b);
    const float2 f = __half22float2(h2);
    const __half2 l2 = __floats2half2_rn(a - f.x, b - f.y);
    h[i] = *reinterpret_cast<const uint32_t*>(&h2);
    l[i] = *reinterpret_cast<const uint32_t*>(&l2);
  }
  hi = make_uint4(h[0], h[1], h[2], h[3]);
  lo = make_uint4(l[0], l[1], l[2], l[3]);
}

// p[0 .. 8), of which n are there (p 16-byte aligned)
__device__ __forceinline__ void load8(const float* p, int n, float (&x)[8]) {
  if (n >= 8) {
    const float4 a = __ldg((const float4*)p), b = __ldg((const float4*)p + 1);
    x[0] = a.x; x[1] = a.y; x[2] = a.z; x[3] = a.w; x[4] = b.x; x[5] = b.y; x[6] = b.z; x[7] = b.w;
  } else {
#pragma unroll
    for (int i = 0; i < 8; ++i) x[i] = i < n ? __ldg(p + i) : 0.0f;
  }
}

// K-major operand: T threads of a block of 256 per row, 8 k-values a piece, the first four pieces of a thread kept in registers
template <int T>
__device__ void split_rows(const PlaneOp& op, int block) {
  constexpr int KEEP = 4;
  __shared__ uint32_t sh[8];
  const int t = threadIdx.x % T, row = block * (256 / T) + (int)threadIdx.x / T;
  const bool live = row < op.rows;
  const float* src = op.src + (int64_t)(live ? row : 0) * op.ld;
  const int pieces = live ? op.num_kb * (IMG_K / 8) : 0;
  float x[KEEP][8];
  uint32_t m = 0;
#pragma unroll
  for (int i = 0; i < KEEP; ++i) {
    const int p = t + i * T;
    if (p < pieces) {
      load8(src + 8 * p, op.K - 8 * p, x[i]);
#pragma unroll
      for (int j = 0; j < 8; ++j) m = max(m, abs_bits(x[i][j]));
    }
  }
  for (int p = t + KEEP * T; p < pieces; p += T) {
    float y[8];
    load8(src + 8 * p, op.K - 8 * p, y);
#pragma unroll
    for (int j = 0; j < 8; ++j) m = max(m, abs_bits(y[j]));
  }
  m = __reduce_max_sync(0xffffffffu, m);
  if (T > 32) {
    const int w = threadIdx.x >> 5;
    if ((threadIdx.x & 31) == 0) sh[w] = m;
    __syncthreads();
#pragma unroll
    for (int i = 0; i < T / 32; ++i) m = max(m, sh[w / (T / 32) * (T / 32) + i]);
  }
  if (!live) return;
  const int s = row_shift(m);
  if (t == 0) op.exps[row] = -s;
  float sc[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) sc[j] = __int_as_float((s + 127) << 23);
  uint16_t* img = op.img + (int64_t)(row / IMG_ROWS) * op.num_kb * (2 * IMG_HALVES) + (row % IMG_ROWS) * IMG_K;
  const bool finite = m < 0x7f800000u;
  auto put = [&](int p, float (&v)[8]) {
    uint4 hi, lo;
    if (finite) leave_out8(op, v, sc, row, 0, 8 * p, 1);
    split8(v, sc, hi, lo);
    uint16_t* d = img + (int64_t)(p >> 3) * (2 * IMG_HALVES) + (p & 7) * 8;
    *(uint4*)d = hi;
    *(uint4*)(d + IMG_HALVES) = lo;
  };
#pragma unroll
  for (int i = 0; i < KEEP; ++i)
    if (t + i * T < pieces) put(t + i * T, x[i]);
  for (int p = t + KEEP * T; p < pieces; p += T) {
    float y[8];
    load8(src + 8 * p, op.K - 8 * p, y);
    put(p, y);
  }
}

// MN-major operand, partial maxima: 128 rows (contiguous in memory) x one chunk of k
__device__ void max_cols(const PlaneOp& op, int block) {
  __shared__ uint32_t sh[8][IMG_ROWS];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int nb = block % ((op.rows + IMG_ROWS - 1) / IMG_ROWS), ch = block / ((op.rows + IMG_ROWS - 1) / IMG_ROWS);
  const int c = nb * IMG_ROWS + 4 * lane;
  const int k0 = ch * op.chunk_k, k1 = min(op.K, k0 + op.chunk_k);
  uint32_t m[4] = {0, 0, 0, 0};
  if (c + 3 < op.rows) {
    const float* p = op.src + c;
#pragma unroll 8
    for (int k = k0 + w; k < k1; k += 8) {
      const float4 v = __ldg((const float4*)(p + (int64_t)k * op.ld));
      m[0] = max(m[0], abs_bits(v.x)); m[1] = max(m[1], abs_bits(v.y)); m[2] = max(m[2], abs_bits(v.z)); m[3] = max(m[3], abs_bits(v.w));
    }
  } else {
    for (int k = k0 + w; k < k1; k += 8)
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (c + j < op.rows) m[j] = max(m[j], abs_bits(__ldg(op.src + (int64_t)k * op.ld + c + j)));
  }
  *(uint4*)&sh[w][4 * lane] = make_uint4(m[0], m[1], m[2], m[3]);
  __syncthreads();
  if (threadIdx.x < IMG_ROWS) {
    uint32_t r = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) r = max(r, sh[i][threadIdx.x]);
    op.part[((int64_t)ch * ((op.rows + IMG_ROWS - 1) / IMG_ROWS) + nb) * IMG_ROWS + threadIdx.x] = r;
  }
}

// MN-major operand: 128 rows x two images' worth of k
__device__ void split_cols(const PlaneOp& op, int block) {
  __shared__ float sh[IMG_ROWS];
  const int nbs = (op.rows + IMG_ROWS - 1) / IMG_ROWS, nb = block % nbs, kp = block / nbs;
  if (threadIdx.x < IMG_ROWS) {
    uint32_t m = 0;
    for (int ch = 0; ch < op.chunks; ++ch) m = max(m, op.part[((int64_t)ch * nbs + nb) * IMG_ROWS + threadIdx.x]);
    const int s = row_shift(m);
    // (a row that is not finite comes out as NaN whatever its other elements: with this scale they are large or zero, and none is listed)
    sh[threadIdx.x] = m < 0x7f800000u ? __int_as_float((s + 127) << 23) : INFINITY;
    if (kp == 0) op.exps[nb * IMG_ROWS + threadIdx.x] = -s;
  }
  __syncthreads();
  const int c8 = 8 * (threadIdx.x & 15), kr = threadIdx.x >> 4;
  const int c = nb * IMG_ROWS + c8, n = op.rows - c;
  float sc[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) sc[j] = sh[c8 + j];
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    const int kb = 2 * kp + q;
    if (kb >= op.num_kb) break;
    uint16_t* img = op.img + ((int64_t)nb * op.num_kb + kb) * (2 * IMG_HALVES) + (c8 >> 6) * (IMG_K * 64) + (c8 & 63);
    float x[4][8];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int k = kb * IMG_K + 16 * i + kr;
      load8(op.src + (int64_t)(k < op.K ? k : 0) * op.ld + (n > 0 ? c : 0), k < op.K ? n : 0, x[i]);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      uint4 hi, lo;
      leave_out8(op, x[i], sc, c, 1, kb * IMG_K + 16 * i + kr, 0);
      split8(x[i], sc, hi, lo);
      uint16_t* d = img + (16 * i + kr) * 64;
      *(uint4*)d = hi;
      *(uint4*)(d + IMG_HALVES) = lo;
    }
  }
}

__device__ void split_rows_any(const PlaneOp& op, int block) {
  if (op.num_kb <= 16) split_rows<32>(op, block);
  else if (op.num_kb <= 64) split_rows<128>(op, block);
  else split_rows<256>(op, block);
}

// first kernel: K-major operands are split, MN-major ones get their maxima; second: MN-major ones are split
__global__ void __launch_bounds__(256, 4) planes_first_kernel(const PlaneOp a, const PlaneOp b) {
  fb_after_previous();
  const bool first = (int)blockIdx.x < a.blocks1;
  const PlaneOp& op = first ? a : b;
  const int block = first ? (int)blockIdx.x : (int)blockIdx.x - a.blocks1;
  if (op.mn_major) max_cols(op, block);
  else split_rows_any(op, block);
}
__global__ void __launch_bounds__(256, 4) planes_second_kernel(const PlaneOp a, const PlaneOp b) {
  fb_after_previous();
  const bool first = (int)blockIdx.x < a.blocks2;
  split_cols(first ? a : b, first ? (int)blockIdx.x : (int)blockIdx.x - a.blocks2);
}

int64_t pad256(int64_t n) { return (n + 255) / 256 * 256; }

struct Sizes {
  int64_t img, exps, part, chunks, chunk_k, left, list, cap;
};
Sizes sizes_of(int64_t rows, int64_t K, int mn_major) {
  const int64_t tiles = (rows + IMG_ROWS - 1) / IMG_ROWS, num_kb = (K + IMG_K - 1) / IMG_K;
  Sizes z;
  z.chunk_k = (K + MAX_CHUNKS - 1) / MAX_CHUNKS < 128 ? 128 : (K + MAX_CHUNKS - 1) / MAX_CHUNKS;
  z.chunks = (K + z.chunk_k - 1) / z.chunk_k;
  z.img = tiles * num_kb * (2 * IMG_HALVES) * 2;
  z.exps = pad256(tiles * IMG_ROWS * 4);
  z.part = mn_major ? pad256(z.chunks * tiles * IMG_ROWS * 4) : 0;
  z.cap = 8 + K / 16384;   // (of N(0, 1) values K / 4,000,000 are expected, of gradients behind a gelu K / 140,000)
  z.left = pad256(tiles * IMG_ROWS * 4);
  z.list = pad256(tiles * IMG_ROWS * z.cap * 8);
  return z;
}

}  // namespace

size_t fb_planes_bytes(const fb_gemm_args& g) {
  const Sizes a = sizes_of(g.M, g.K, g.a_mn_major), b = sizes_of(g.N, g.K, g.b_mn_major);
  return fb_planes_zero_bytes(g) + (size_t)(a.img + a.exps + a.part + a.list + b.img + b.exps + b.part + b.list);
}
size_t fb_planes_zero_bytes(const fb_gemm_args& g) {
  return (size_t)(256 + sizes_of(g.M, g.K, g.a_mn_major).left + sizes_of(g.N, g.K, g.b_mn_major).left);
}

int32_t fb_planes_split(cudaStream_t stream, const fb_gemm_args& g, void* mem, fb_planes* out) {
  PlaneOp op[2];
  char *z0 = (char*)mem, *p = z0 + fb_planes_zero_bytes(g);
  int64_t blocks1 = 0, blocks2 = 0;
  out->over = (int32_t*)z0; z0 += 256;
  for (int i = 0; i < 2; ++i) {
    PlaneOp& o = op[i];
    const int64_t rows = i == 0 ? g.M : g.N, ld = i == 0 ? g.lda : g.ldb;
    o.src = i == 0 ? g.A : g.B;
    o.ld = ld;
    o.mn_major = i == 0 ? g.a_mn_major : g.b_mn_major;
    const Sizes z = sizes_of(rows, g.K, o.mn_major);
    o.rows = (int)rows;
    o.K = (int)g.K;
    o.num_kb = (int)((g.K + IMG_K - 1) / IMG_K);
    o.img = (uint16_t*)p; p += z.img;
    o.exps = (int32_t*)p; p += z.exps;
    o.part = (uint32_t*)p; p += z.part;
    o.list = (int2*)p; p += z.list;
    o.left = (int32_t*)z0; z0 += z.left;
    o.cap = (int)z.cap;
    o.over = out->over;
    o.least = fb_planes_least(g.K);
    out->left[i] = o.left;
    out->list[i] = o.list;
    out->cap = o.cap;
    o.chunks = (int)z.chunks;
    o.chunk_k = (int)z.chunk_k;
    const int64_t tiles = (rows + IMG_ROWS - 1) / IMG_ROWS;
    const int per = o.num_kb <= 16 ? 8 : o.num_kb <= 64 ? 2 : 1;   // rows per block (split_rows_any)
    const int64_t n1 = o.mn_major ? tiles * z.chunks : (rows + per - 1) / per;
    const int64_t n2 = o.mn_major ? tiles * ((o.num_kb + 1) / 2) : 0;
    o.blocks1 = (int)n1;
    o.blocks2 = (int)n2;
    blocks1 += n1;
    blocks2 += n2;
    out->img[i] = o.img;
    out->exps[i] = o.exps;
    out->rows[i] = tiles * o.num_kb * 2 * IMG_ROWS;
  }
  if (blocks1 > 0x7fffffff || blocks2 > 0x7fffffff) return fb_fail(FB_ERR_UNSUPPORTED, "gemm: operands too large to split");
  fb_launch(planes_first_kernel, (unsigned)blocks1, 256, 0, stream, op[0], op[1]);
  FB_LAUNCH_CHECK();
  if (blocks2 > 0) {
    fb_launch(planes_second_kernel, (unsigned)blocks2, 256, 0, stream, op[0], op[1]);
    FB_LAUNCH_CHECK();
  }
  return FB_OK;
}
