// The bf16 entry points of the Dense path (Flux.bf16, src/functor.jl:274): matmul and Dense forward / backward with
// BFloat16 storage for weights, activations and gradients, fp32 accumulation on the tensor cores (gemm_bf16.cu).
//
// Row-major views of Julia's column-major arrays, as in dense.cu:
//   forward   Y[n][out]    = X[n][in]    * Wm[in][out]        (A K-major,  B MN-major, bias along out)
//   dX        dX[n][in]    = D[n][out]   * Wm[in][out]^T      (A K-major,  B K-major)
//   dW        dWm[in][out] = X[n][in]^T  * D[n][out]          (A MN-major, B MN-major)
#include <cuda_bf16.h>

#include "common.cuh"

namespace {

__device__ __forceinline__ float bf2f(uint16_t v) { return __uint_as_float((uint32_t)v << 16); }
__device__ __forceinline__ uint16_t f2bf(float v) {
  const __nv_bfloat16 b = __float2bfloat16_rn(v);
  return *reinterpret_cast<const uint16_t*>(&b);
}

// W consecutive bf16 values (16 bytes at W = 8)
template <int W>
__device__ __forceinline__ void ld_bf(const uint16_t* p, float (&v)[W]) {
  if constexpr (W == 8) {
    const uint4 w = *(const uint4*)p;
    const uint32_t u[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      v[2 * e] = __uint_as_float(u[e] << 16);
      v[2 * e + 1] = __uint_as_float(u[e] & 0xffff0000u);
    }
  } else {
    v[0] = bf2f(*p);
  }
}

// delta = dy .* act'(.) (bf16) and per-block partial column sums of delta (fp32): block (x: 32 W columns, y: row group), a warp a
// row.  Bound: HBM and, for the gelu flavours, their derivative: 4096 columns x 2048 rows with gelu 23.6 -> 18.3 us, of 1000 columns
// without an activation 5.0 -> 3.8 (one value a thread and load before).
template <int W, int KIND>
__global__ void __launch_bounds__(256)
act_bwd_colsum_bf16_kernel(int act, const uint16_t* __restrict__ dy, const uint16_t* __restrict__ y, const uint16_t* __restrict__ z,
                           uint16_t* __restrict__ delta, float* __restrict__ part, int64_t rows, int64_t cols, int64_t rpb) {
  constexpr int U = 2;
  __shared__ float sh[8][32 * W];
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const int64_t col = ((int64_t)blockIdx.x * 32 + tx) * W;
  const int64_t r0 = (int64_t)blockIdx.y * rpb, r1 = (r0 + rpb < rows) ? r0 + rpb : rows;
  const bool from_z = KIND == 2 && (act == FB_ACT_GELU_TANH || act == FB_ACT_GELU_ERF);
  const uint16_t* src = from_z ? z : y;
  float s[W];
#pragma unroll
  for (int e = 0; e < W; ++e) s[e] = 0.0f;
  if (col < cols) {
    for (int64_t r = r0 + ty; r < r1; r += 8 * U) {
      float d[U][W], a[U][W];
#pragma unroll
      for (int u = 0; u < U; ++u)
        if (r + 8 * u < r1) {
          ld_bf<W>(dy + (r + 8 * u) * cols + col, d[u]);
          if (KIND != 0) ld_bf<W>(src + (r + 8 * u) * cols + col, a[u]);
        }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        if (r + 8 * u >= r1) break;
        if (KIND != 0) {
          uint16_t q[W];
#pragma unroll
          for (int e = 0; e < W; ++e) {
            if (KIND == 1) d[u][e] *= a[u][e] > 0.0f ? 1.0f : 0.0f;
            else d[u][e] *= from_z ? fb_act_grad_z(act, a[u][e]) : fb_act_grad_y(act, a[u][e]);
            q[e] = f2bf(d[u][e]);
            d[u][e] = bf2f(q[e]);          // the bias gradient sums what the GEMMs will read
          }
          uint16_t* o = delta + (r + 8 * u) * cols + col;
          if constexpr (W == 8) {
            uint32_t w[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) w[e] = (uint32_t)q[2 * e] | ((uint32_t)q[2 * e + 1] << 16);
            *(uint4*)o = make_uint4(w[0], w[1], w[2], w[3]);
          } else {
            *o = q[0];
          }
        }
#pragma unroll
        for (int e = 0; e < W; ++e) s[e] += d[u][e];
      }
    }
  }
  if (part == nullptr) return;
#pragma unroll
  for (int e = 0; e < W; ++e) sh[ty][tx * W + e] = s[e];
  __syncthreads();
  for (int k = threadIdx.x; k < 32 * W; k += 256) {
    const int64_t c = (int64_t)blockIdx.x * 32 * W + k;
    if (c >= cols) break;
    float t = 0.0f;
#pragma unroll
    for (int i = 0; i < 8; ++i) t += sh[i][k];
    part[(int64_t)blockIdx.y * cols + c] = t;
  }
}

// a block: 32 columns, eight groups of partial rows at a time
__global__ void __launch_bounds__(256) colsum_parts_bf16_kernel(const float* __restrict__ part, uint16_t* __restrict__ out, int64_t groups, int64_t cols) {
  __shared__ float sh[8][33];
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const int64_t c = (int64_t)blockIdx.x * 32 + tx;
  float s = 0.0f;
  if (c < cols) {
#pragma unroll 4
    for (int64_t g = ty; g < groups; g += 8) s += part[g * cols + c];
  }
  sh[ty][tx] = s;
  __syncthreads();
  if (ty != 0 || c >= cols) return;
#pragma unroll
  for (int i = 1; i < 8; ++i) s += sh[i][tx];
  out[c] = f2bf(s);
}

__global__ void __launch_bounds__(256) axpy_bf16_kernel(float alpha, const uint16_t* __restrict__ x, uint16_t* __restrict__ y, int64_t count) {
  for (int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x; i < count; i += (int64_t)gridDim.x * 256)
    y[i] = f2bf(fmaf(alpha, bf2f(x[i]), bf2f(y[i])));
}

}  // namespace

FB_API int32_t fb_axpy_bf16(fb_ctx* ctx, void* stream, float alpha, const uint16_t* x, uint16_t* y, int64_t count) {
  FB_CHECK_CTX(ctx);
  FB_REQUIRE(count >= 0, FB_ERR_INVALID_ARG, "fb_axpy_bf16: negative count");
  if (count == 0) return FB_OK;
  FB_REQUIRE(x && y, FB_ERR_INVALID_ARG, "fb_axpy_bf16: NULL pointer");
  int64_t blocks = (count + 255) / 256;
  if (blocks > (int64_t)ctx->sm_count * 16) blocks = (int64_t)ctx->sm_count * 16;
  axpy_bf16_kernel<<<(unsigned)blocks, 256, 0, (cudaStream_t)stream>>>(alpha, x, y, count);
  FB_LAUNCH_CHECK();
  return FB_OK;
}

FB_API int32_t fb_gemm_bf16(fb_ctx* ctx, void* stream, int32_t transa, int32_t transb, int64_t m, int64_t n, int64_t k,
                            const uint16_t* A, int64_t lda, const uint16_t* B, int64_t ldb, void* C, int64_t ldc,
                            int32_t accumulate, int32_t c_is_f32) {
  FB_CHECK_CTX(ctx);
  FB_REQUIRE(m >= 0 && n >= 0 && k >= 0, FB_ERR_SHAPE, "fb_gemm_bf16: negative dimension");
  FB_REQUIRE((transa == 0 || transa == 1) && (transb == 0 || transb == 1), FB_ERR_INVALID_ARG, "fb_gemm_bf16: trans flags must be 0 or 1");
  if (m == 0 || n == 0) return FB_OK;
  FB_REQUIRE(k >= 1, FB_ERR_SHAPE, "fb_gemm_bf16: k must be at least 1");
  FB_REQUIRE(A && B && C, FB_ERR_INVALID_ARG, "fb_gemm_bf16: NULL pointer");
  FB_REQUIRE(lda >= (transa ? k : m) && ldb >= (transb ? n : k) && ldc >= m, FB_ERR_SHAPE, "fb_gemm_bf16: leading dimension too small");
  // column-major C[m,n] is the row-major C'[n][m] = op(B)^T * op(A)^T
  fb_gemm_bf16_args a;
  a.A = B; a.lda = ldb; a.a_mn_major = transb ? 1 : 0;
  a.B = A; a.ldb = lda; a.b_mn_major = transa ? 0 : 1;
  a.C = C; a.ldc = ldc; a.Z = nullptr; a.bias_n = nullptr;
  a.M = n; a.N = m; a.K = k; a.act = FB_ACT_IDENTITY; a.accumulate = accumulate ? 1 : 0; a.out_f32 = c_is_f32 ? 1 : 0;
  return fb_gemm_bf16_launch(ctx, (cudaStream_t)stream, a);
}

FB_API int32_t fb_dense_fwd_bf16(fb_ctx* ctx, void* stream, int32_t act, const uint16_t* W, const uint16_t* b, const uint16_t* x,
                                 uint16_t* y, uint16_t* z, int64_t out_dim, int64_t in_dim, int64_t n) {
  FB_CHECK_CTX(ctx);
  FB_REQUIRE(out_dim >= 1 && in_dim >= 1 && n >= 0, FB_ERR_SHAPE, "fb_dense_fwd_bf16: bad shape out=%lld in=%lld n=%lld",
             (long long)out_dim, (long long)in_dim, (long long)n);
  FB_REQUIRE(fb_act_valid(act), FB_ERR_INVALID_ARG, "fb_dense_fwd_bf16: unknown activation %d", act);
  if (n == 0) return FB_OK;
  FB_REQUIRE(W && x && y, FB_ERR_INVALID_ARG, "fb_dense_fwd_bf16: NULL pointer");
  fb_gemm_bf16_args a;
  a.A = x; a.lda = in_dim; a.a_mn_major = 0;
  a.B = W; a.ldb = out_dim; a.b_mn_major = 1;
  a.C = y; a.ldc = out_dim; a.Z = z; a.bias_n = b;
  a.M = n; a.N = out_dim; a.K = in_dim; a.act = act; a.accumulate = 0; a.out_f32 = 0;
  return fb_gemm_bf16_launch(ctx, (cudaStream_t)stream, a);
}

FB_API int32_t fb_dense_bwd_bf16(fb_ctx* ctx, void* stream_, int32_t act, const uint16_t* W, const uint16_t* x, const uint16_t* y,
                                 const uint16_t* z, const uint16_t* dy, uint16_t* delta, uint16_t* dW, uint16_t* db, uint16_t* dx,
                                 int64_t out_dim, int64_t in_dim, int64_t n) {
  FB_CHECK_CTX(ctx);
  cudaStream_t stream = (cudaStream_t)stream_;
  FB_REQUIRE(out_dim >= 1 && in_dim >= 1 && n >= 1, FB_ERR_SHAPE, "fb_dense_bwd_bf16: bad shape out=%lld in=%lld n=%lld",
             (long long)out_dim, (long long)in_dim, (long long)n);
  FB_REQUIRE(fb_act_valid(act), FB_ERR_INVALID_ARG, "fb_dense_bwd_bf16: unknown activation %d", act);
  FB_REQUIRE(W && x && dy && dW, FB_ERR_INVALID_ARG, "fb_dense_bwd_bf16: NULL pointer");
  const bool need_delta = (act != FB_ACT_IDENTITY);
  if (need_delta) {
    FB_REQUIRE(delta != nullptr, FB_ERR_INVALID_ARG, "fb_dense_bwd_bf16: delta scratch is required for a non-identity activation");
    if (fb_act_needs_z(act)) FB_REQUIRE(z != nullptr, FB_ERR_INVALID_ARG, "fb_dense_bwd_bf16: the gelu activations need the saved pre-activation z");
    else FB_REQUIRE(y != nullptr, FB_ERR_INVALID_ARG, "fb_dense_bwd_bf16: the forward output y is required");
  }
  if (need_delta || db != nullptr) {
    const uint16_t* src = fb_act_needs_z(act) ? z : y;
    const bool vec = out_dim % 8 == 0 && fb_aligned16(dy) && (!need_delta || (fb_aligned16(src) && fb_aligned16(delta)));
    const int64_t per = 32 * (vec ? 8 : 1), gx = (out_dim + per - 1) / per;
    int64_t gy = ((int64_t)ctx->sm_count * 8 + gx - 1) / gx;
    if (gy > (n + 15) / 16) gy = (n + 15) / 16;
    if (gy < 1) gy = 1;
    if (gy > 65535) gy = 65535;
    const int64_t rpb = (n + gy - 1) / gy;
    gy = (n + rpb - 1) / rpb;
    float* part = nullptr;
    if (db != nullptr) {
      part = (float*)fb_scratch(ctx, stream, (size_t)(gy * out_dim) * sizeof(float));
      if (!part) return FB_ERR_ALLOC;
    }
    fb_act_kind(act, [&](auto k) {
      const dim3 grid((unsigned)gx, (unsigned)gy);
      if (vec) act_bwd_colsum_bf16_kernel<8, k.value><<<grid, 256, 0, stream>>>(act, dy, y, z, delta, part, n, out_dim, rpb);
      else act_bwd_colsum_bf16_kernel<1, k.value><<<grid, 256, 0, stream>>>(act, dy, y, z, delta, part, n, out_dim, rpb);
    });
    FB_LAUNCH_CHECK();
    if (db != nullptr) {
      colsum_parts_bf16_kernel<<<(unsigned)((out_dim + 31) / 32), 256, 0, stream>>>(part, db, gy, out_dim);
      FB_LAUNCH_CHECK();
    }
  }
  const uint16_t* D = need_delta ? delta : dy;
  fb_gemm_bf16_args a;
  a.Z = nullptr; a.bias_n = nullptr; a.act = FB_ACT_IDENTITY; a.accumulate = 0; a.out_f32 = 0;
  a.A = x; a.lda = in_dim; a.a_mn_major = 1;
  a.B = D; a.ldb = out_dim; a.b_mn_major = 1;
  a.C = dW; a.ldc = out_dim; a.M = in_dim; a.N = out_dim; a.K = n;
  int32_t st = fb_gemm_bf16_launch(ctx, stream, a);
  if (st != FB_OK) return st;
  if (dx != nullptr) {
    a.A = D; a.lda = out_dim; a.a_mn_major = 0;
    a.B = W; a.ldb = out_dim; a.b_mn_major = 0;
    a.C = dx; a.ldc = in_dim; a.M = n; a.N = in_dim; a.K = out_dim;
    st = fb_gemm_bf16_launch(ctx, stream, a);
  }
  return st;
}
