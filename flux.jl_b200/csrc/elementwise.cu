// Element-wise helpers, the loss kernels and the multi-tensor Adam step (all memory-bound).
#include <cuda_bf16.h>

#include "common.cuh"
#include "tc_common.cuh"

namespace {

constexpr int EW_THREADS = 256;

unsigned ew_grid(const fb_ctx* ctx, int64_t items) {
  int64_t blocks = (items + EW_THREADS - 1) / EW_THREADS;
  const int64_t cap = (int64_t)ctx->sm_count * 32;
  if (blocks > cap) blocks = cap;
  if (blocks < 1) blocks = 1;
  return (unsigned)blocks;
}

__global__ void __launch_bounds__(EW_THREADS)
scale_kernel(const float* __restrict__ x, float alpha, float* __restrict__ y, int64_t count, int vec) {
  fb_after_previous();
  const int64_t tid = (int64_t)blockIdx.x * EW_THREADS + threadIdx.x, stride = (int64_t)gridDim.x * EW_THREADS;
  if (vec) {
    const float4* x4 = (const float4*)x;
    float4* y4 = (float4*)y;
    for (int64_t i = tid; i < (count >> 2); i += stride) {
      float4 v = __ldcs(x4 + i);
      v.x *= alpha; v.y *= alpha; v.z *= alpha; v.w *= alpha;
      __stcs(y4 + i, v);
    }
    for (int64_t i = (count & ~int64_t(3)) + tid; i < count; i += stride) y[i] = alpha * x[i];
  } else {
    for (int64_t i = tid; i < count; i += stride) y[i] = alpha * x[i];
  }
}

__global__ void __launch_bounds__(EW_THREADS)
axpy_kernel(float alpha, const float* __restrict__ x, float* __restrict__ y, int64_t count, int vec) {
  fb_after_previous();
  const int64_t tid = (int64_t)blockIdx.x * EW_THREADS + threadIdx.x, stride = (int64_t)gridDim.x * EW_THREADS;
  if (vec) {
    const float4* x4 = (const float4*)x;
    float4* y4 = (float4*)y;
    for (int64_t i = tid; i < (count >> 2); i += stride) {
      const float4 a = __ldcs(x4 + i);
      float4 b = y4[i];
      b.x = fmaf(alpha, a.x, b.x); b.y = fmaf(alpha, a.y, b.y); b.z = fmaf(alpha, a.z, b.z); b.w = fmaf(alpha, a.w, b.w);
      y4[i] = b;
    }
    for (int64_t i = (count & ~int64_t(3)) + tid; i < count; i += stride) y[i] = fmaf(alpha, x[i], y[i]);
  } else {
    for (int64_t i = tid; i < count; i += stride) y[i] = fmaf(alpha, x[i], y[i]);
  }
}

__global__ void __launch_bounds__(EW_THREADS)
cast_f32_bf16_kernel(const float* __restrict__ x, uint16_t* __restrict__ y, int64_t count, int vec) {
  fb_after_previous();
  const int64_t tid = (int64_t)blockIdx.x * EW_THREADS + threadIdx.x, stride = (int64_t)gridDim.x * EW_THREADS;
  // eight values a thread where both arrays allow it (16.8 M values: 21 -> 14.7 us, 2 M values 9.2 -> 4.7)
  int64_t done = 0;
  if (vec) {
    done = count & ~int64_t(7);
    for (int64_t i = tid; i < (count >> 3); i += stride) {
      const float4 a = __ldcs((const float4*)x + 2 * i), b = __ldcs((const float4*)x + 2 * i + 1);
      const float v[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
      uint32_t w[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) w[e] = (uint32_t)fb_bf16_bits(v[2 * e]) | ((uint32_t)fb_bf16_bits(v[2 * e + 1]) << 16);
      ((uint4*)y)[i] = make_uint4(w[0], w[1], w[2], w[3]);
    }
  }
  for (int64_t i = done + tid; i < count; i += stride) y[i] = fb_bf16_bits(x[i]);
}

__global__ void __launch_bounds__(EW_THREADS)
cast_bf16_f32_kernel(const uint16_t* __restrict__ x, float* __restrict__ y, int64_t count, int vec) {
  fb_after_previous();
  const int64_t tid = (int64_t)blockIdx.x * EW_THREADS + threadIdx.x, stride = (int64_t)gridDim.x * EW_THREADS;
  int64_t done = 0;
  if (vec) {
    done = count & ~int64_t(7);
    for (int64_t i = tid; i < (count >> 3); i += stride) {
      const uint4 w = __ldcs((const uint4*)x + i);
      ((float4*)y)[2 * i] = make_float4(__uint_as_float(w.x << 16), __uint_as_float(w.x & 0xffff0000u), __uint_as_float(w.y << 16), __uint_as_float(w.y & 0xffff0000u));
      ((float4*)y)[2 * i + 1] = make_float4(__uint_as_float(w.z << 16), __uint_as_float(w.z & 0xffff0000u), __uint_as_float(w.w << 16), __uint_as_float(w.w & 0xffff0000u));
    }
  }
  for (int64_t i = done + tid; i < count; i += stride) y[i] = __uint_as_float((uint32_t)x[i] << 16);
}

// ------------------------------------------------------------------------------- sum of squares ---
__global__ void __launch_bounds__(EW_THREADS)
sumsq_partial_kernel(const float* __restrict__ x, int64_t count, float* __restrict__ part, int vec, int square) {
  fb_after_previous();
  __shared__ float sh[32];
  const int64_t tid = (int64_t)blockIdx.x * EW_THREADS + threadIdx.x, stride = (int64_t)gridDim.x * EW_THREADS;
  float s = 0.0f;
  if (vec) {
    const float4* x4 = (const float4*)x;
    for (int64_t i = tid; i < (count >> 2); i += stride) {
      const float4 v = __ldcs(x4 + i);
      s += square ? (v.x * v.x + v.y * v.y) + (v.z * v.z + v.w * v.w) : (v.x + v.y) + (v.z + v.w);
    }
    for (int64_t i = (count & ~int64_t(3)) + tid; i < count; i += stride) s += square ? x[i] * x[i] : x[i];
  } else {
    for (int64_t i = tid; i < count; i += stride) s += square ? x[i] * x[i] : x[i];
  }
  s = fb_block_sum(s, sh);
  if (threadIdx.x == 0) part[blockIdx.x] = s;
}

// out[0] = scale * sum(part[0..m))   (one block; fixed order -> run-to-run deterministic)
__global__ void __launch_bounds__(1024)
final_sum_kernel(const float* __restrict__ part, int64_t m, float scale, float* __restrict__ out) {
  fb_after_previous();
  fb_let_next_start();
  __shared__ float sh[32];
  float s = 0.0f;
  for (int64_t i = threadIdx.x; i < m; i += 1024) s += part[i];
  s = fb_block_sum(s, sh);
  if (threadIdx.x == 0) out[0] = s * scale;
}

// ------------------------------------------------------------------------ logit cross-entropy ---
// One warp per sample (column of Julia yhat[c, n] = row of the [n][c] buffer).
template <bool LABELS>
__global__ void __launch_bounds__(128)
xent_kernel(const float* __restrict__ yhat, const int32_t* __restrict__ labels, const float* __restrict__ ydense,
            float* __restrict__ loss_part, float* __restrict__ dyhat, int64_t c, int64_t n, float gscale) {
  fb_after_previous();
  fb_let_next_start();
  const int lane = threadIdx.x & 31;
  const int64_t row = (int64_t)blockIdx.x * 4 + (threadIdx.x >> 5);
  if (row >= n) return;
  const float* z = yhat + row * c;
  float mx = -INFINITY;
  for (int64_t j = lane; j < c; j += 32) mx = fmaxf(mx, z[j]);
  mx = fb_warp_max(mx);
  float se = 0.0f, sy = 0.0f, syz = 0.0f;
  for (int64_t j = lane; j < c; j += 32) {
    const float zj = z[j];
    se += expf(zj - mx);
    if (!LABELS) {
      const float yj = ydense[row * c + j];
      sy += yj;
      syz += yj * zj;
    }
  }
  se = fb_warp_sum(se);
  const float lse = mx + logf(se);
  int64_t lab = 0;
  if (LABELS) {
    lab = (int64_t)labels[row] - 1;  // labels are 1-based, as onehotbatch(labels, 1:c)
    sy = 1.0f;
    syz = (lab >= 0 && lab < c) ? z[lab] : 0.0f;
  } else {
    sy = fb_warp_sum(sy);
    syz = fb_warp_sum(syz);
  }
  // -sum_j y_j (z_j - lse) = lse * sum(y) - sum(y z)
  if (lane == 0) loss_part[row] = lse * sy - syz;
  if (dyhat != nullptr) {
    float* d = dyhat + row * c;
    for (int64_t j = lane; j < c; j += 32) {
      const float p = expf(z[j] - lse);
      const float yj = LABELS ? (j == lab ? 1.0f : 0.0f) : ydense[row * c + j];
      d[j] = (p * sy - yj) * gscale;
    }
  }
}

// ------------------------------------------------------------------------------------- Adam ---
constexpr int ADAM_MAX_TENSORS = 32;
constexpr int ADAM_CHUNK = 8192;  // elements per block

struct AdamTable {
  float* w[ADAM_MAX_TENSORS];
  const float* g[ADAM_MAX_TENSORS];
  float* m[ADAM_MAX_TENSORS];
  float* v[ADAM_MAX_TENSORS];
  long long count[ADAM_MAX_TENSORS];
  int block_start[ADAM_MAX_TENSORS + 1];
  int ntensors;
};

// Two shapes of one kernel.  The plain one (256 threads) streams at the HBM roofline when it has the GPU to itself.
// The side one (128 threads of at most 32 registers) fits on an SM beside a resident GEMM CTA - one warp per
// register-file partition - so an update enqueued on the communication stream does not wait for the reverse sweep's
// GEMM to end; alone it reaches about 70 % of the plain one's bandwidth.
constexpr int ADAM_SIDE_THREADS = 128;
template <int ADAM_THREADS, int MIN_BLOCKS>
__global__ void __launch_bounds__(ADAM_THREADS, MIN_BLOCKS)
adam_kernel(const __grid_constant__ AdamTable tab, float eta, float beta1, float beta2, float eps, float inv_c1,
            float inv_c2, float grad_scale, const float* __restrict__ bt_dev, const float* __restrict__ guard) {
  fb_after_previous();
  // device-resident step state (used when the step is replayed from a CUDA graph): the running beta powers
  // and an optional guard scalar (the loss) whose non-finite value skips the update
  if (guard != nullptr && !isfinite(__ldg(guard))) return;
  if (bt_dev != nullptr) {
    inv_c1 = 1.0f / (1.0f - __ldg(bt_dev));
    inv_c2 = 1.0f / (1.0f - __ldg(bt_dev + 1));
  }
  int t = 0;
  while (t + 1 < tab.ntensors && (int)blockIdx.x >= tab.block_start[t + 1]) ++t;
  const int64_t begin = (int64_t)(blockIdx.x - tab.block_start[t]) * ADAM_CHUNK;
  const int64_t count = tab.count[t];
  int64_t end = begin + ADAM_CHUNK;
  if (end > count) end = count;
  float* w = tab.w[t];
  const float* g = tab.g[t];
  float* m = tab.m[t];
  float* v = tab.v[t];
  const float omb1 = 1.0f - beta1, omb2 = 1.0f - beta2;
  const bool vec = ((reinterpret_cast<uintptr_t>(w) | reinterpret_cast<uintptr_t>(g) | reinterpret_cast<uintptr_t>(m) |
                     reinterpret_cast<uintptr_t>(v)) & 15u) == 0;
  if (vec) {
    const int64_t e4 = begin + ((end - begin) & ~int64_t(3));
    for (int64_t i = begin + 4 * threadIdx.x; i < e4; i += 4 * ADAM_THREADS) {
      float4 gv = __ldcs((const float4*)(g + i));
      float4 mv = *(const float4*)(m + i), vv = *(const float4*)(v + i), wv = *(const float4*)(w + i);
      float* gp = &gv.x; float* mp = &mv.x; float* vp = &vv.x; float* wp = &wv.x;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const float gk = gp[k] * grad_scale;
        mp[k] = beta1 * mp[k] + omb1 * gk;
        vp[k] = beta2 * vp[k] + omb2 * gk * gk;
        wp[k] -= mp[k] * inv_c1 / (sqrtf(vp[k] * inv_c2) + eps) * eta;
      }
      *(float4*)(m + i) = mv;
      *(float4*)(v + i) = vv;
      *(float4*)(w + i) = wv;
    }
    for (int64_t i = e4 + threadIdx.x; i < end; i += ADAM_THREADS) {
      const float gk = g[i] * grad_scale;
      const float mk = beta1 * m[i] + omb1 * gk, vk = beta2 * v[i] + omb2 * gk * gk;
      m[i] = mk; v[i] = vk;
      w[i] -= mk * inv_c1 / (sqrtf(vk * inv_c2) + eps) * eta;
    }
  } else {
    for (int64_t i = begin + threadIdx.x; i < end; i += ADAM_THREADS) {
      const float gk = g[i] * grad_scale;
      const float mk = beta1 * m[i] + omb1 * gk, vk = beta2 * v[i] + omb2 * gk * gk;
      m[i] = mk; v[i] = vk;
      w[i] -= mk * inv_c1 / (sqrtf(vk * inv_c2) + eps) * eta;
    }
  }
}

// The update of bf16 parameters: the rule runs on the Float32 master copy with the bf16 gradient widened in registers, and
// the rounded parameter is written in the same pass.  Bound by memory: 28 bytes a parameter; as three passes (gradient to
// Float32, update, rounding) it moved 40.  54.5 M parameters in 14 leaves: 400 us in 15 launches -> 235 us in one (6490 GB/s).
struct AdamLowTable {
  AdamTable t;                          // g unused
  const uint16_t* g[ADAM_MAX_TENSORS];
  uint16_t* p[ADAM_MAX_TENSORS];
};

__device__ __forceinline__ uint16_t adam_round(float w) {
  const __nv_bfloat16 b = __float2bfloat16_rn(w);
  return *reinterpret_cast<const uint16_t*>(&b);
}

__global__ void __launch_bounds__(256)
adam_bf16_kernel(const __grid_constant__ AdamLowTable tab, float eta, float beta1, float beta2, float eps, float inv_c1, float inv_c2,
                 float grad_scale) {
  fb_after_previous();
  int t = 0;
  while (t + 1 < tab.t.ntensors && (int)blockIdx.x >= tab.t.block_start[t + 1]) ++t;
  const int64_t begin = (int64_t)(blockIdx.x - tab.t.block_start[t]) * ADAM_CHUNK;
  const int64_t count = tab.t.count[t];
  const int64_t end = begin + ADAM_CHUNK > count ? count : begin + ADAM_CHUNK;
  float *w = tab.t.w[t], *m = tab.t.m[t], *v = tab.t.v[t];
  const uint16_t* g = tab.g[t];
  uint16_t* p = tab.p[t];
  const float omb1 = 1.0f - beta1, omb2 = 1.0f - beta2;
  auto rule = [&](float gk, float& mk, float& vk, float& wk) {
    gk *= grad_scale;
    mk = beta1 * mk + omb1 * gk;
    vk = beta2 * vk + omb2 * gk * gk;
    wk -= mk * inv_c1 / (sqrtf(vk * inv_c2) + eps) * eta;
  };
  const bool vec = ((reinterpret_cast<uintptr_t>(w) | reinterpret_cast<uintptr_t>(m) | reinterpret_cast<uintptr_t>(v)) & 15u) == 0 &&
                   ((reinterpret_cast<uintptr_t>(g) | reinterpret_cast<uintptr_t>(p)) & 7u) == 0;
  int64_t i0 = begin;
  if (vec) {
    i0 = begin + ((end - begin) & ~int64_t(3));
    for (int64_t i = begin + 4 * threadIdx.x; i < i0; i += 4 * 256) {
      const uint2 gw = __ldcs((const uint2*)(g + i));
      const float gv[4] = {__uint_as_float(gw.x << 16), __uint_as_float(gw.x & 0xffff0000u), __uint_as_float(gw.y << 16),
                           __uint_as_float(gw.y & 0xffff0000u)};
      float4 mv = *(const float4*)(m + i), vv = *(const float4*)(v + i), wv = *(const float4*)(w + i);
      float *mp = &mv.x, *vp = &vv.x, *wp = &wv.x;
      uint32_t r[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        rule(gv[k], mp[k], vp[k], wp[k]);
        r[k] = adam_round(wp[k]);
      }
      *(float4*)(m + i) = mv;
      *(float4*)(v + i) = vv;
      *(float4*)(w + i) = wv;
      *(uint2*)(p + i) = make_uint2(r[0] | (r[1] << 16), r[2] | (r[3] << 16));
    }
  }
  for (int64_t i = i0 + threadIdx.x; i < end; i += 256) {
    float mk = m[i], vk = v[i], wk = w[i];
    rule(__uint_as_float((uint32_t)g[i] << 16), mk, vk, wk);
    m[i] = mk; v[i] = vk; w[i] = wk;
    p[i] = adam_round(wk);
  }
}

// ------------------------------------------------- activation backward + bias-gradient column sum ---
// delta[r][j] = dy[r][j] * act'(.) ; part[blockIdx.y][j] = sum over this block's rows of delta[r][j], or (CL) part[j] = the sum over
// all rows: the up to 8 row groups of a column block are a cluster.
// Block = 32 x 8 threads; thread (tx, ty) owns VEC consecutive columns, U rows in flight.
template <int VEC, bool CL>
__global__ void __launch_bounds__(256)
act_bwd_colsum_kernel(int act, const float* __restrict__ dy, const float* __restrict__ y, const float* __restrict__ z,
                      float* __restrict__ delta, float* __restrict__ part, int64_t rows, int64_t cols,
                      int64_t rows_per_block) {
  fb_after_previous();
  fb_let_next_start();
  constexpr int U = CL ? 4 : 1;
  __shared__ float sh[8][32 * VEC + 1];
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const int64_t col0 = ((int64_t)blockIdx.x * 32 + tx) * VEC;
  const int64_t r_begin = (int64_t)blockIdx.y * rows_per_block;
  int64_t r_end = r_begin + rows_per_block;
  if (r_end > rows) r_end = rows;
  const bool use_z = (act == FB_ACT_GELU_TANH || act == FB_ACT_GELU_ERF);
  const float* src = use_z ? z : y;
  float acc[VEC];
#pragma unroll
  for (int k = 0; k < VEC; ++k) acc[k] = 0.0f;
  if (col0 < cols) {
    for (int64_t r = r_begin + ty; r < r_end; r += 8 * U) {
      float d[U][VEC], s[U][VEC];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int64_t off = (r + 8 * u) * cols + col0;
        if (r + 8 * u >= r_end) continue;
        if constexpr (VEC == 4) {
          const float4 dv = __ldcs((const float4*)(dy + off));
          d[u][0] = dv.x; d[u][1] = dv.y; d[u][2] = dv.z; d[u][3] = dv.w;
          if (act != FB_ACT_IDENTITY) {
            const float4 sv = __ldcs((const float4*)(src + off));
            s[u][0] = sv.x; s[u][1] = sv.y; s[u][2] = sv.z; s[u][3] = sv.w;
          }
        } else {
          d[u][0] = dy[off];
          if (act != FB_ACT_IDENTITY) s[u][0] = src[off];
        }
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        if (r + 8 * u >= r_end) break;
        const int64_t off = (r + 8 * u) * cols + col0;
        if (act != FB_ACT_IDENTITY)
#pragma unroll
          for (int k = 0; k < VEC; ++k) d[u][k] *= use_z ? fb_act_grad_z(act, s[u][k]) : fb_act_grad_y(act, s[u][k]);
        if (delta != nullptr) {
          if constexpr (VEC == 4) __stcs((float4*)(delta + off), make_float4(d[u][0], d[u][1], d[u][2], d[u][3]));
          else delta[off] = d[u][0];
        }
#pragma unroll
        for (int k = 0; k < VEC; ++k) acc[k] += d[u][k];
      }
    }
  }
  if (part == nullptr) return;   // (uniform)
#pragma unroll
  for (int k = 0; k < VEC; ++k) sh[ty][tx * VEC + k] = acc[k];
  __syncthreads();
  if (CL) {
    if (threadIdx.x < 32 * VEC) {
      float s = 0.0f;
#pragma unroll
      for (int i = 0; i < 8; ++i) s += sh[i][threadIdx.x];
      sh[0][threadIdx.x] = s;
    }
    cluster_column_sums(sh[0], 32 * VEC, part + (int64_t)blockIdx.x * (32 * VEC), cols - (int64_t)blockIdx.x * (32 * VEC), gridDim.y);
  } else if (ty == 0 && col0 < cols) {
#pragma unroll
    for (int k = 0; k < VEC; ++k) {
      float s = 0.0f;
#pragma unroll
      for (int i = 0; i < 8; ++i) s += sh[i][tx * VEC + k];
      part[(int64_t)blockIdx.y * cols + col0 + k] = s;
    }
  }
}

}  // namespace

__global__ void fb_colreduce2_kernel(const float* part_a, const float* part_b, float* out_a, float* out_b,
                                     int64_t groups, int64_t d);

int32_t fb_act_bwd_colsum(fb_ctx* ctx, cudaStream_t stream, int act, const float* dy, const float* y,
                          const float* z, float* delta, float* db, int64_t rows, int64_t cols) {
  const bool need_delta = (act != FB_ACT_IDENTITY);
  if (!need_delta && db == nullptr) return FB_OK;
  if (need_delta) {
    FB_REQUIRE(delta != nullptr, FB_ERR_INVALID_ARG, "dense backward: delta scratch is required for a non-identity activation");
    if (fb_act_needs_z(act)) FB_REQUIRE(z != nullptr, FB_ERR_INVALID_ARG, "dense backward: the gelu activations need the saved pre-activation z");
    else FB_REQUIRE(y != nullptr, FB_ERR_INVALID_ARG, "dense backward: the forward output y is required");
  }
  const float* src = fb_act_needs_z(act) ? z : y;
  const bool vec = (cols % 4 == 0) && fb_aligned16(dy) && (!need_delta || (fb_aligned16(delta) && fb_aligned16(src)));
  const int V = vec ? 4 : 1;
  const int64_t gx = (cols + 32 * V - 1) / (32 * V);
  // Up to 512 rows: eight row groups, one cluster, no second kernel.  More rows need more blocks than that, and their partial sums
  // are added up by a kernel of its own (1024 rows of 512 with gelu: 4.4 and 5.1 us, as one cluster 10.7).
  const bool one = db != nullptr && rows <= 512 && gx <= 0xfffffff;
  int64_t gy = one ? 8 : ((int64_t)ctx->sm_count * 8 + gx - 1) / gx;
  if (gy > (rows + 7) / 8) gy = (rows + 7) / 8;
  if (gy < 1) gy = 1;
  if (gy > 65535) gy = 65535;
  const int64_t rpb = (rows + gy - 1) / gy;
  gy = (rows + rpb - 1) / rpb;
  dim3 grid((unsigned)gx, (unsigned)gy);
  float* dout = need_delta ? delta : nullptr;
  if (one) {
    cudaLaunchConfig_t lc;
    memset(&lc, 0, sizeof(lc));
    lc.gridDim = grid;
    lc.blockDim = dim3(256, 1, 1);
    lc.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = attr[0].val.clusterDim.z = 1;
    attr[0].val.clusterDim.y = (unsigned)gy;
    lc.attrs = attr;
    lc.numAttrs = 1;
    FB_CUDA(cudaLaunchKernelEx(&lc, vec ? act_bwd_colsum_kernel<4, true> : act_bwd_colsum_kernel<1, true>, act, dy, y, z, dout, db, rows, cols, rpb));
    FB_LAUNCH_CHECK();
    return FB_OK;
  }
  float* part = nullptr;
  if (db != nullptr) {
    part = (float*)fb_scratch(ctx, stream, (size_t)(gy * cols) * sizeof(float));
    if (!part) return FB_ERR_ALLOC;
  }
  if (vec) fb_launch(act_bwd_colsum_kernel<4, false>, grid, 256, 0, stream, act, dy, y, z, dout, part, rows, cols, rpb);
  else fb_launch(act_bwd_colsum_kernel<1, false>, grid, 256, 0, stream, act, dy, y, z, dout, part, rows, cols, rpb);
  FB_LAUNCH_CHECK();
  if (db != nullptr) {
    fb_launch(fb_colreduce2_kernel, (unsigned)((cols + 31) / 32), 256, 0, stream, part, nullptr, db, nullptr, gy, cols);
    FB_LAUNCH_CHECK();
  }
  return FB_OK;
}

FB_API int32_t fb_scale(fb_ctx* ctx, void* stream, const float* x, float alpha, float* y, int64_t count) {
  FB_CHECK_CTX(ctx);
  FB_REQUIRE(count >= 0, FB_ERR_INVALID_ARG, "fb_scale: negative count");
  if (count == 0) return FB_OK;
  FB_REQUIRE(x && y, FB_ERR_INVALID_ARG, "fb_scale: NULL pointer");
  const int vec = fb_aligned16(x) && fb_aligned16(y);
  fb_launch(scale_kernel, ew_grid(ctx, vec ? (count + 3) / 4 : count), EW_THREADS, 0, (cudaStream_t)stream, x, alpha, y, count, vec);
  FB_LAUNCH_CHECK();
  return FB_OK;
}

__global__ void __launch_bounds__(256) fill_kernel(float* __restrict__ x, float value, int64_t count) {
  fb_after_previous();
  for (int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x; i < count; i += (int64_t)gridDim.x * 256) x[i] = value;
}

FB_API int32_t fb_fill(fb_ctx* ctx, void* stream, float* x, float value, int64_t count) {
  FB_CHECK_CTX(ctx);
  FB_REQUIRE(count >= 0, FB_ERR_INVALID_ARG, "fb_fill: negative count");
  if (count == 0) return FB_OK;
  FB_REQUIRE(x, FB_ERR_INVALID_ARG, "fb_fill: NULL pointer");
  int64_t blocks = (count + 255) / 256;
  if (blocks > (int64_t)ctx->sm_count * 32) blocks = (int64_t)ctx->sm_count * 32;
  fb_launch(fill_kernel, (unsigned)blocks, 256, 0, (cudaStream_t)stream, x, value, count);
  FB_LAUNCH_CHECK();
  return FB_OK;
}

// One thread stores the GPU's nanosecond timer: a stream-ordered time mark that also works inside a captured graph
// (where events cannot be timed).
__global__ void timestamp_kernel(uint64_t* out) {
  fb_after_previous();
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  *out = t;
}

int32_t fb_side_kernels_prepare_elementwise() {
  FB_CUDA(cudaFuncSetAttribute(adam_kernel<ADAM_SIDE_THREADS, 2048 / ADAM_SIDE_THREADS>, cudaFuncAttributePreferredSharedMemoryCarveout,
                               cudaSharedmemCarveoutMaxShared));
  FB_CUDA(cudaFuncSetAttribute(timestamp_kernel, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared));
  return FB_OK;
}

FB_API int32_t fb_timestamp(fb_ctx* ctx, void* stream, uint64_t* out_dev) {
  FB_CHECK_CTX(ctx);
  FB_REQUIRE(out_dev, FB_ERR_INVALID_ARG, "fb_timestamp: NULL pointer");
  fb_launch(timestamp_kernel, 1, 1, 0, (cudaStream_t)stream, out_dev);
  FB_LAUNCH_CHECK();
  return FB_OK;
}

FB_API int32_t fb_axpy(fb_ctx* ctx, void* stream, float alpha, const float* x, float* y, int64_t count) {
  FB_CHECK_CTX(ctx);
  FB_REQUIRE(count >= 0, FB_ERR_INVALID_ARG, "fb_axpy: negative count");
  if (count == 0) return FB_OK;
  FB_REQUIRE(x && y, FB_ERR_INVALID_ARG, "fb_axpy: NULL pointer");
  const int vec = fb_aligned16(x) && fb_aligned16(y);
  fb_launch(axpy_kernel, ew_grid(ctx, vec ? (count + 3) / 4 : count), EW_THREADS, 0, (cudaStream_t)stream, alpha, x, y, count, vec);
  FB_LAUNCH_CHECK();
  return FB_OK;
}

__global__ void __launch_bounds__(EW_THREADS)
round_bf16_kernel(const float* __restrict__ x, float* __restrict__ y, int64_t count) {
  fb_after_previous();
  const int64_t tid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = tid; i < count; i += stride) y[i] = __uint_as_float((uint32_t)fb_bf16_bits(x[i]) << 16);
}

FB_API int32_t fb_round_bf16(fb_ctx* ctx, void* stream, const float* x, float* y, int64_t count) {
  FB_CHECK_CTX(ctx);
  FB_REQUIRE(count >= 0, FB_ERR_INVALID_ARG, "fb_round_bf16: negative count");
  if (count == 0) return FB_OK;
  FB_REQUIRE(x && y, FB_ERR_INVALID_ARG, "fb_round_bf16: NULL pointer");
  fb_launch(round_bf16_kernel, ew_grid(ctx, count), EW_THREADS, 0, (cudaStream_t)stream, x, y, count);
  FB_LAUNCH_CHECK();
  return FB_OK;
}

// out = a + b in Float32, each term Float32 or BFloat16 (out may be one of them): a sum of two arrays in one pass
template <bool AB, bool BB>
__global__ void __launch_bounds__(EW_THREADS)
add_kernel(const void* a, const void* b, float* out, int64_t count, int vec) {
  fb_after_previous();
  const int64_t tid = (int64_t)blockIdx.x * EW_THREADS + threadIdx.x, stride = (int64_t)gridDim.x * EW_THREADS;
  auto four = [](const void* p, bool low, int64_t i, float (&v)[4]) {
    if (low) {
      const uint2 w = ((const uint2*)p)[i];
      v[0] = __uint_as_float(w.x << 16); v[1] = __uint_as_float(w.x & 0xffff0000u);
      v[2] = __uint_as_float(w.y << 16); v[3] = __uint_as_float(w.y & 0xffff0000u);
    } else {
      const float4 q = ((const float4*)p)[i];
      v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
    }
  };
  auto one = [](const void* p, bool low, int64_t i) {
    return low ? __uint_as_float((uint32_t)((const uint16_t*)p)[i] << 16) : ((const float*)p)[i];
  };
  int64_t done = 0;
  if (vec) {
    done = count & ~int64_t(3);
    for (int64_t i = tid; i < (count >> 2); i += stride) {
      float x[4], y[4];
      four(a, AB, i, x);
      four(b, BB, i, y);
      ((float4*)out)[i] = make_float4(x[0] + y[0], x[1] + y[1], x[2] + y[2], x[3] + y[3]);
    }
  }
  for (int64_t i = done + tid; i < count; i += stride) out[i] = one(a, AB, i) + one(b, BB, i);
}

FB_API int32_t fb_add_mixed(fb_ctx* ctx, void* stream_, const void* a, int32_t a_bf16, const void* b, int32_t b_bf16, float* out, int64_t count) {
  FB_CHECK_CTX(ctx);
  FB_REQUIRE(count >= 0, FB_ERR_INVALID_ARG, "fb_add_mixed: negative count");
  if (count == 0) return FB_OK;
  FB_REQUIRE(a && b && out, FB_ERR_INVALID_ARG, "fb_add_mixed: NULL pointer");
  cudaStream_t stream = (cudaStream_t)stream_;
  const int vec = fb_aligned16(a) && fb_aligned16(b) && fb_aligned16(out);
  const unsigned grid = ew_grid(ctx, vec ? (count + 3) / 4 : count);
  if (a_bf16 && b_bf16) fb_launch(add_kernel<true, true>, grid, EW_THREADS, 0, stream, a, b, out, count, vec);
  else if (a_bf16) fb_launch(add_kernel<true, false>, grid, EW_THREADS, 0, stream, a, b, out, count, vec);
  else if (b_bf16) fb_launch(add_kernel<false, true>, grid, EW_THREADS, 0, stream, a, b, out, count, vec);
  else fb_launch(add_kernel<false, false>, grid, EW_THREADS, 0, stream, a, b, out, count, vec);
  FB_LAUNCH_CHECK();
  return FB_OK;
}

FB_API int32_t fb_cast_f32_bf16(fb_ctx* ctx, void* stream, const float* x, uint16_t* y, int64_t count) {
  FB_CHECK_CTX(ctx);
  FB_REQUIRE(count >= 0, FB_ERR_INVALID_ARG, "fb_cast_f32_bf16: negative count");
  if (count == 0) return FB_OK;
  FB_REQUIRE(x && y, FB_ERR_INVALID_ARG, "fb_cast_f32_bf16: NULL pointer");
  const int vec = fb_aligned16(x) && fb_aligned16(y);
  fb_launch(cast_f32_bf16_kernel, ew_grid(ctx, vec ? (count + 7) / 8 : count), EW_THREADS, 0, (cudaStream_t)stream, x, y, count, vec);
  FB_LAUNCH_CHECK();
  return FB_OK;
}

FB_API int32_t fb_cast_bf16_f32(fb_ctx* ctx, void* stream, const uint16_t* x, float* y, int64_t count) {
  FB_CHECK_CTX(ctx);
  FB_REQUIRE(count >= 0, FB_ERR_INVALID_ARG, "fb_cast_bf16_f32: negative count");
  if (count == 0) return FB_OK;
  FB_REQUIRE(x && y, FB_ERR_INVALID_ARG, "fb_cast_bf16_f32: NULL pointer");
  const int vec = fb_aligned16(x) && fb_aligned16(y);
  fb_launch(cast_bf16_f32_kernel, ew_grid(ctx, vec ? (count + 7) / 8 : count), EW_THREADS, 0, (cudaStream_t)stream, x, y, count, vec);
  FB_LAUNCH_CHECK();
  return FB_OK;
}

static int32_t sum_common(fb_ctx* ctx, cudaStream_t stream, const float* x, int64_t count, float* out, int square,
                          const char* fn) {
  FB_REQUIRE(count >= 0 && out, FB_ERR_INVALID_ARG, "%s: bad arguments", fn);
  if (count == 0) {
    FB_CUDA(cudaMemsetAsync(out, 0, sizeof(float), stream));
    return FB_OK;
  }
  FB_REQUIRE(x, FB_ERR_INVALID_ARG, "%s: NULL pointer", fn);
  const int vec = fb_aligned16(x);
  int64_t blocks = ((vec ? count / 4 : count) + EW_THREADS - 1) / EW_THREADS;
  const int64_t cap = (int64_t)ctx->sm_count * 8;
  if (blocks > cap) blocks = cap;
  if (blocks < 1) blocks = 1;
  float* part = (float*)fb_scratch(ctx, stream, (size_t)blocks * sizeof(float));
  if (!part) return FB_ERR_ALLOC;
  fb_launch(sumsq_partial_kernel, (unsigned)blocks, EW_THREADS, 0, stream, x, count, part, vec, square);
  FB_LAUNCH_CHECK();
  fb_launch(final_sum_kernel, 1, 1024, 0, stream, part, blocks, 1.0f, out);
  FB_LAUNCH_CHECK();
  return FB_OK;
}

FB_API int32_t fb_sumsq(fb_ctx* ctx, void* stream, const float* x, int64_t count, float* out) {
  FB_CHECK_CTX(ctx);
  return sum_common(ctx, (cudaStream_t)stream, x, count, out, 1, "fb_sumsq");
}

FB_API int32_t fb_sum(fb_ctx* ctx, void* stream, const float* x, int64_t count, float* out) {
  FB_CHECK_CTX(ctx);
  return sum_common(ctx, (cudaStream_t)stream, x, count, out, 0, "fb_sum");
}

static int32_t xent_common(fb_ctx* ctx, cudaStream_t stream, const float* yhat, const int32_t* labels, const float* y,
                           float* loss, float* dyhat, int64_t c, int64_t n, float dloss, const char* fn) {
  FB_REQUIRE(c >= 1 && n >= 1, FB_ERR_SHAPE, "%s: bad shape c=%lld n=%lld", fn, (long long)c, (long long)n);
  FB_REQUIRE(yhat && loss && (labels || y), FB_ERR_INVALID_ARG, "%s: NULL pointer", fn);
  float* part = (float*)fb_scratch(ctx, stream, (size_t)n * sizeof(float));
  if (!part) return FB_ERR_ALLOC;
  const unsigned grid = (unsigned)((n + 3) / 4);
  const float gscale = dloss / (float)n;
  if (labels) fb_launch(xent_kernel<true>, grid, 128, 0, stream, yhat, labels, nullptr, part, dyhat, c, n, gscale);
  else fb_launch(xent_kernel<false>, grid, 128, 0, stream, yhat, nullptr, y, part, dyhat, c, n, gscale);
  FB_LAUNCH_CHECK();
  fb_launch(final_sum_kernel, 1, 1024, 0, stream, part, n, 1.0f / (float)n, loss);
  FB_LAUNCH_CHECK();
  return FB_OK;
}

FB_API int32_t fb_logitcrossentropy_labels(fb_ctx* ctx, void* stream, const float* yhat, const int32_t* labels,
                                           float* loss, float* dyhat, int64_t c, int64_t n, float dloss) {
  FB_CHECK_CTX(ctx);
  FB_REQUIRE(labels, FB_ERR_INVALID_ARG, "fb_logitcrossentropy_labels: labels is NULL");
  return xent_common(ctx, (cudaStream_t)stream, yhat, labels, nullptr, loss, dyhat, c, n, dloss, "fb_logitcrossentropy_labels");
}

FB_API int32_t fb_logitcrossentropy_dense(fb_ctx* ctx, void* stream, const float* yhat, const float* y, float* loss,
                                          float* dyhat, int64_t c, int64_t n, float dloss) {
  FB_CHECK_CTX(ctx);
  FB_REQUIRE(y, FB_ERR_INVALID_ARG, "fb_logitcrossentropy_dense: y is NULL");
  return xent_common(ctx, (cudaStream_t)stream, yhat, nullptr, y, loss, dyhat, c, n, dloss, "fb_logitcrossentropy_dense");
}

static int32_t adam_common(fb_ctx* ctx, cudaStream_t stream, int32_t ntensors, float* const* w_host,
                           const float* const* g_host, float* const* m_host, float* const* v_host,
                           const int64_t* counts_host, float eta, float beta1, float beta2, float eps, float b1t,
                           float b2t, float grad_scale, const float* bt_dev, const float* guard, bool side = false);

FB_API int32_t fb_adam_step(fb_ctx* ctx, void* stream_, int32_t ntensors, float* const* w_host,
                            const float* const* g_host, float* const* m_host, float* const* v_host,
                            const int64_t* counts_host, float eta, float beta1, float beta2, float eps, float b1t,
                            float b2t, float grad_scale) {
  FB_CHECK_CTX(ctx);
  return adam_common(ctx, (cudaStream_t)stream_, ntensors, w_host, g_host, m_host, v_host, counts_host, eta, beta1, beta2, eps,
                     b1t, b2t, grad_scale, nullptr, nullptr);
}

FB_API int32_t fb_adam_step_bf16(fb_ctx* ctx, void* stream_, int32_t ntensors, uint16_t* const* p_host, float* const* w_host,
                                 const uint16_t* const* g_host, float* const* m_host, float* const* v_host, const int64_t* counts_host,
                                 float eta, float beta1, float beta2, float eps, float b1t, float b2t, float grad_scale) {
  FB_CHECK_CTX(ctx);
  FB_REQUIRE(ntensors >= 0, FB_ERR_INVALID_ARG, "fb_adam_step_bf16: negative tensor count");
  if (ntensors == 0) return FB_OK;
  FB_REQUIRE(p_host && w_host && g_host && m_host && v_host && counts_host, FB_ERR_INVALID_ARG, "fb_adam_step_bf16: NULL table");
  for (int i = 0; i < ntensors; ++i) {
    FB_REQUIRE(counts_host[i] >= 0 && counts_host[i] < (int64_t)ADAM_CHUNK << 24, FB_ERR_INVALID_ARG,
               "fb_adam_step_bf16: bad element count for leaf %d", i);
    FB_REQUIRE(counts_host[i] == 0 || (p_host[i] && w_host[i] && g_host[i] && m_host[i] && v_host[i]), FB_ERR_INVALID_ARG,
               "fb_adam_step_bf16: NULL pointer for leaf %d", i);
  }
  const float inv_c1 = 1.0f / (1.0f - b1t), inv_c2 = 1.0f / (1.0f - b2t);
  int done = 0;
  while (done < ntensors) {
    AdamLowTable tab;
    memset(&tab, 0, sizeof(tab));
    int k = 0, blocks = 0;
    for (; done < ntensors && k < ADAM_MAX_TENSORS; ++done) {
      if (counts_host[done] == 0) continue;
      tab.t.w[k] = w_host[done]; tab.t.m[k] = m_host[done]; tab.t.v[k] = v_host[done];
      tab.g[k] = g_host[done]; tab.p[k] = p_host[done];
      tab.t.count[k] = counts_host[done];
      tab.t.block_start[k++] = blocks;
      blocks += (int)((counts_host[done] + ADAM_CHUNK - 1) / ADAM_CHUNK);   // 32 leaves of < 2^24 blocks
    }
    if (k == 0) continue;
    tab.t.block_start[k] = blocks;
    tab.t.ntensors = k;
    fb_launch(adam_bf16_kernel, (unsigned)blocks, 256, 0, (cudaStream_t)stream_, tab, eta, beta1, beta2, eps, inv_c1, inv_c2, grad_scale);
    FB_LAUNCH_CHECK();
  }
  return FB_OK;
}

FB_API int32_t fb_adam_step_dev(fb_ctx* ctx, void* stream_, int32_t ntensors, float* const* w_host,
                                const float* const* g_host, float* const* m_host, float* const* v_host,
                                const int64_t* counts_host, float eta, float beta1, float beta2, float eps,
                                const float* bt_dev, const float* guard_dev, float grad_scale) {
  FB_CHECK_CTX(ctx);
  FB_REQUIRE(bt_dev != nullptr, FB_ERR_INVALID_ARG, "fb_adam_step_dev: bt_dev is NULL");
  return adam_common(ctx, (cudaStream_t)stream_, ntensors, w_host, g_host, m_host, v_host, counts_host, eta, beta1, beta2, eps,
                     0.0f, 0.0f, grad_scale, bt_dev, guard_dev);
}

FB_API int32_t fb_adam_block_dev(fb_ctx* ctx, void* stream_, float* w, const float* g, float* m, float* v, int64_t count, float eta,
                                 float beta1, float beta2, float eps, const float* bt_dev, const float* guard_dev, float grad_scale) {
  FB_CHECK_CTX(ctx);
  FB_REQUIRE(bt_dev != nullptr, FB_ERR_INVALID_ARG, "fb_adam_block_dev: bt_dev is NULL");
  return adam_common(ctx, (cudaStream_t)stream_, 1, &w, &g, &m, &v, &count, eta, beta1, beta2, eps, 0.0f, 0.0f, grad_scale, bt_dev,
                     guard_dev, true);
}

__global__ void adam_advance_kernel(float* __restrict__ bt, float beta1, float beta2, const float* __restrict__ guard) {
  fb_after_previous();
  fb_let_next_start();
  if (guard != nullptr && !isfinite(*guard)) return;
  bt[0] *= beta1;
  bt[1] *= beta2;
}

FB_API int32_t fb_adam_advance(fb_ctx* ctx, void* stream_, float* bt_dev, float beta1, float beta2, const float* guard_dev) {
  FB_CHECK_CTX(ctx);
  FB_REQUIRE(bt_dev != nullptr, FB_ERR_INVALID_ARG, "fb_adam_advance: bt_dev is NULL");
  fb_launch(adam_advance_kernel, 1, 1, 0, (cudaStream_t)stream_, bt_dev, beta1, beta2, guard_dev);
  FB_LAUNCH_CHECK();
  return FB_OK;
}

static int32_t adam_common(fb_ctx* ctx, cudaStream_t stream, int32_t ntensors, float* const* w_host,
                           const float* const* g_host, float* const* m_host, float* const* v_host,
                           const int64_t* counts_host, float eta, float beta1, float beta2, float eps, float b1t,
                           float b2t, float grad_scale, const float* bt_dev, const float* guard, bool side) {
  FB_REQUIRE(ntensors >= 0, FB_ERR_INVALID_ARG, "fb_adam_step: negative tensor count");
  if (ntensors == 0) return FB_OK;
  FB_REQUIRE(w_host && g_host && m_host && v_host && counts_host, FB_ERR_INVALID_ARG, "fb_adam_step: NULL table");
  // bias corrections in the parameter eltype (Float32), as the rule computes them
  const float inv_c1 = 1.0f / (1.0f - b1t), inv_c2 = 1.0f / (1.0f - b2t);
  int done = 0;
  while (done < ntensors) {
    AdamTable tab;
    memset(&tab, 0, sizeof(tab));
    int k = 0, blocks = 0;
    while (done < ntensors && k < ADAM_MAX_TENSORS) {
      const int64_t cnt = counts_host[done];
      FB_REQUIRE(cnt >= 0, FB_ERR_INVALID_ARG, "fb_adam_step: negative element count for leaf %d", done);
      if (cnt > 0) {
        FB_REQUIRE(w_host[done] && g_host[done] && m_host[done] && v_host[done], FB_ERR_INVALID_ARG,
                   "fb_adam_step: NULL pointer for leaf %d", done);
        const int64_t nb = (cnt + ADAM_CHUNK - 1) / ADAM_CHUNK;
        if ((int64_t)blocks + nb > 0x3fffffff) break;
        tab.w[k] = w_host[done]; tab.g[k] = g_host[done]; tab.m[k] = m_host[done]; tab.v[k] = v_host[done];
        tab.count[k] = cnt;
        tab.block_start[k] = blocks;
        blocks += (int)nb;
        ++k;
      }
      ++done;
    }
    if (k == 0) continue;
    tab.block_start[k] = blocks;
    tab.ntensors = k;
    if (side)
      adam_kernel<ADAM_SIDE_THREADS, 2048 / ADAM_SIDE_THREADS><<<(unsigned)blocks, ADAM_SIDE_THREADS, 0, stream>>>(
          tab, eta, beta1, beta2, eps, inv_c1, inv_c2, grad_scale, bt_dev, guard);
    else
      fb_launch(adam_kernel<EW_THREADS, 1>, (unsigned)blocks, EW_THREADS, 0, stream, tab, eta, beta1, beta2, eps, inv_c1, inv_c2, grad_scale,
                                                                              bt_dev, guard);
    FB_LAUNCH_CHECK();
  }
  return FB_OK;
}
