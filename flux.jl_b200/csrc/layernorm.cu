// LayerNorm forward / backward (memory-bound).
//
// Data layout: x is [n][d] row-major (Julia x[d, n]); statistics run over the d contiguous floats of a
// row.  Forward: one read of x, one write of y (the row lives in registers between the two reductions).
// Backward: one read each of x and dy, one write of dx; dgamma / dbeta are accumulated per thread in
// registers across the rows a block owns and reduced in a second, small kernel from per-block partials.
// Where only dgamma / dbeta are wanted the backward pass is a sum over columns and needs no row sums at all.
//
// Rows of up to 1024 features belong to one warp each (no block barriers, every load of a row in flight at once), longer ones to
// a block.  Rows that are no whole number of aligned float4 are read float by float, up to 8192 features in registers too.
#include "common.cuh"
#include "tc_common.cuh"

namespace {

constexpr int LN_THREADS = 256;

__device__ __forceinline__ float4 ld_stream(const float4* p) { return __ldcs(p); }
__device__ __forceinline__ void st_stream(float4* p, float4 v) { __stcs(p, v); }

// Two block-wide sums at once.  sh must hold 64 floats.
__device__ __forceinline__ void block_sum2(float& a, float& b, float* sh) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  a = fb_warp_sum(a);
  b = fb_warp_sum(b);
  __syncthreads();
  if (lane == 0) { sh[w] = a; sh[32 + w] = b; }
  __syncthreads();
  float ra = (lane < nw) ? sh[lane] : 0.0f;
  float rb = (lane < nw) ? sh[32 + lane] : 0.0f;
  a = fb_warp_sum(ra);
  b = fb_warp_sum(rb);
}

// ------------------------------------------------------------------ forward, row in registers ---
template <int V>
__global__ void __launch_bounds__(LN_THREADS)
ln_fwd_vec_kernel(const float4* __restrict__ x, const float4* __restrict__ gamma,
                  const float4* __restrict__ beta, float4* __restrict__ y, float* __restrict__ mean,
                  float* __restrict__ rstd, int d4, int64_t n, float eps, int act) {
  fb_after_previous();
  __shared__ float sh[64];
  const float inv_d = 1.0f / (4.0f * (float)d4);
  for (int64_t row = blockIdx.x; row < n; row += gridDim.x) {
    const float4* xr = x + row * d4;
    float4 v[V];
    float s = 0.0f;
#pragma unroll
    for (int i = 0; i < V; ++i) {
      const int c = threadIdx.x + i * LN_THREADS;
      if (c < d4) {
        v[i] = ld_stream(xr + c);
        s += (v[i].x + v[i].y) + (v[i].z + v[i].w);
      } else {
        v[i] = make_float4(0.f, 0.f, 0.f, 0.f);
      }
    }
    const float mu = __fmul_rn(fb_block_sum(s, sh), inv_d);
    float q = 0.0f;
#pragma unroll
    for (int i = 0; i < V; ++i) {
      const int c = threadIdx.x + i * LN_THREADS;
      if (c < d4) {
        const float a = v[i].x - mu, b = v[i].y - mu, cc = v[i].z - mu, dd = v[i].w - mu;
        q += (a * a + b * b) + (cc * cc + dd * dd);
      }
    }
    const float var = __fmul_rn(fb_block_sum(q, sh), inv_d);
    const float rs = rsqrtf(var + eps);
    if (threadIdx.x == 0) {
      mean[row] = mu;
      rstd[row] = rs;
    }
    float4* yr = y + row * d4;
#pragma unroll
    for (int i = 0; i < V; ++i) {
      const int c = threadIdx.x + i * LN_THREADS;
      if (c < d4) {
        float4 o;
        o.x = (v[i].x - mu) * rs; o.y = (v[i].y - mu) * rs; o.z = (v[i].z - mu) * rs; o.w = (v[i].w - mu) * rs;
        if (gamma != nullptr) {
          const float4 g = __ldg(gamma + c), b = __ldg(beta + c);
          o.x = fmaf(o.x, g.x, b.x); o.y = fmaf(o.y, g.y, b.y); o.z = fmaf(o.z, g.z, b.z); o.w = fmaf(o.w, g.w, b.w);
        }
        if (act != FB_ACT_IDENTITY) {
          o.x = fb_act_apply(act, o.x); o.y = fb_act_apply(act, o.y);
          o.z = fb_act_apply(act, o.z); o.w = fb_act_apply(act, o.w);
        }
        st_stream(yr + c, o);
      }
    }
  }
}

// ------------------------------------------------- rows in registers, any alignment ---
// T threads per row (a warp, or the block of 256), V pieces of W = VEC ? 4 : 1 floats each.  Bound: HBM and the latency of a row's
// loads and sums.  Forward, from a cold cache: 1001 features x 3000 rows 16 -> 13 us (a block per row that read it three times),
// 1024 x 16384 34 -> 24, 64 x 16384 24 -> 4 (a block per row of 16 pieces), 8191 x 2000 55 -> 37.
template <int W>
__device__ __forceinline__ void ld_piece(const float* p, float* v) {
  if (W == 4) {
    const float4 q = *(const float4*)p;
    v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
  } else {
    v[0] = *p;
  }
}
template <int W>
__device__ __forceinline__ void st_piece(float* p, const float* v) {
  if (W == 4) *(float4*)p = make_float4(v[0], v[1], v[2], v[3]);
  else *p = v[0];
}
template <int T>
__device__ __forceinline__ float row_sum(float v, float* sh) {
  return T == 32 ? fb_warp_sum(v) : fb_block_sum(v, sh);
}
// (x + y) + (z + w) of a piece of four, of its square, of its product with another
__device__ __forceinline__ float sum4(const float* v) { return (v[0] + v[1]) + (v[2] + v[3]); }
__device__ __forceinline__ float dot4(const float* a, const float* b) { return fmaf(a[0], b[0], a[1] * b[1]) + fmaf(a[2], b[2], a[3] * b[3]); }

// M sums over a row from the sums of its fours (four neighbouring values each), in the order in which a block of 256 threads with a four
// each adds them: thread by thread within a warp's 32 fours, then the (up to eight) sums of 32.  A row's statistics so have
// the same bits whichever kernel reads it, and the BFloat16 roundings behind them do not depend on the kernel.
//
// A block: four i of thread t is t + 256 i of the row.  A warp, pieces of P fours: piece i of a lane is lane + 32 i, so that for P = 2 a
// lane's fours are neighbours and lane bit 4 is the lowest bit of the 32 that they belong to.  Every exchange halves a lane's
// fours while there are several (12 shuffles a sum for eight, not 43).
template <int V, int P, int T, int M>
__device__ __forceinline__ void row_sums(float (&p)[M][V * P], float (&out)[M], float* sh) {
  if constexpr (T != 32) {
    static_assert(P == 1, "fours of a block");
#pragma unroll
    for (int k = 0; k < M; ++k) {
      out[k] = 0.0f;
#pragma unroll
      for (int i = 0; i < V; ++i) out[k] += p[k][i];
    }
    if constexpr (M == 1) out[0] = fb_block_sum(out[0], sh);
    else block_sum2(out[0], out[1], sh);
  } else {
    static_assert(V * P <= 8 && (V & (V - 1)) == 0, "fours of a lane");
    const int lane = threadIdx.x & 31;
    constexpr int TOP = P == 2 ? 8 : 16;   // the lane bit whose partner's four lies 16 fours away
    int o = TOP;
#pragma unroll
    for (int m = V * P / 2; m > 0; m /= 2, o /= 2) {
      const bool upper = (lane & o) != 0;
#pragma unroll
      for (int i = 0; i < m; ++i)
#pragma unroll
        for (int k = 0; k < M; ++k) {
          const float give = upper ? p[k][i] : p[k][i + m], keep = upper ? p[k][i + m] : p[k][i];
          p[k][i] = keep + __shfl_xor_sync(0xffffffffu, give, o);
        }
    }
    auto add = [&](int b) {
#pragma unroll
      for (int k = 0; k < M; ++k) out[k] += __shfl_xor_sync(0xffffffffu, out[k], b);
    };
#pragma unroll
    for (int k = 0; k < M; ++k) out[k] = p[k][0];
    for (; o > 0; o /= 2) add(o);
    if (P == 2) add(TOP / V);               // the two fours of a piece
#pragma unroll
    for (int m = V / 2, b = TOP; m > 0; m /= 2, b /= 2) add(b);
    if (P == 2) add(16);
  }
}

// mean and 1 / std of a row of d values in pieces of P fours
template <int V, int P, int T>
__device__ __forceinline__ void row_stats(const float (&v)[V][4 * P], int t, int d, float inv_d, float eps, float* sh, float& mu, float& rs) {
  float p[1][V * P], s[1];
#pragma unroll
  for (int i = 0; i < V; ++i)
#pragma unroll
    for (int h = 0; h < P; ++h) p[0][i * P + h] = (t + i * T) * 4 * P < d ? sum4(v[i] + 4 * h) : 0.0f;
  row_sums<V, P, T>(p, s, sh);
  mu = __fmul_rn(s[0], inv_d);   // (products that end a sum are not fused into what follows: one result in every kernel)
#pragma unroll
  for (int i = 0; i < V; ++i)
#pragma unroll
    for (int h = 0; h < P; ++h) {
      float a[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) a[e] = v[i][4 * h + e] - mu;
      p[0][i * P + h] = (t + i * T) * 4 * P < d ? dot4(a, a) : 0.0f;
    }
  row_sums<V, P, T>(p, s, sh);
  rs = rsqrtf(__fmul_rn(s[0], inv_d) + eps);
}

template <int V, int T, bool VEC, int ACT>
__global__ void __launch_bounds__(LN_THREADS, VEC && V == 8 ? 2 : VEC && V == 4 ? 3 : 1)
ln_fwd_rows_kernel(const float* __restrict__ x, const float* __restrict__ gamma, const float* __restrict__ beta,
                   float* __restrict__ y, float* __restrict__ mean, float* __restrict__ rstd, int d, int64_t n, float eps, int act) {
  fb_after_previous();
  constexpr int W = VEC ? 4 : 1;
  __shared__ float sh[64];
  const int t = threadIdx.x % T;
  const float inv_d = 1.0f / (float)d;
  for (int64_t row = (int64_t)blockIdx.x * (LN_THREADS / T) + threadIdx.x / T; row < n; row += (int64_t)gridDim.x * (LN_THREADS / T)) {
    const float* xr = x + row * d;
    float v[V][W];
#pragma unroll
    for (int i = 0; i < V; ++i) {
      const int c = (t + i * T) * W;
      if (c < d) ld_piece<W>(xr + c, v[i]);
    }
    float mu, rs;
    if constexpr (VEC) {
      row_stats<V, 1, T>(v, t, d, inv_d, eps, sh, mu, rs);
    } else {
      float s = 0.0f;
#pragma unroll
      for (int i = 0; i < V; ++i)
        if (t + i * T < d) s += v[i][0];
      mu = row_sum<T>(s, sh) * inv_d;
      float q = 0.0f;
#pragma unroll
      for (int i = 0; i < V; ++i)
        if (t + i * T < d) { const float a = v[i][0] - mu; q = fmaf(a, a, q); }
      rs = rsqrtf(row_sum<T>(q, sh) * inv_d + eps);
    }
    if (t == 0) {
      mean[row] = mu;
      rstd[row] = rs;
    }
    float* yr = y + row * d;
    constexpr int B = V < 8 ? V : 8;   // pieces whose gamma and beta are loaded together
#pragma unroll
    for (int i0 = 0; i0 < V; i0 += B) {
      float g[B][W], b[B][W];
      if (gamma != nullptr) {
#pragma unroll
        for (int k = 0; k < B; ++k) {
          const int c = (t + (i0 + k) * T) * W;
          if (c < d) {
            ld_piece<W>(gamma + c, g[k]);
            ld_piece<W>(beta + c, b[k]);
          }
        }
      }
#pragma unroll
      for (int k = 0; k < B; ++k) {
        const int c = (t + (i0 + k) * T) * W;
        float o[W];
#pragma unroll
        for (int e = 0; e < W; ++e) {
          o[e] = (v[i0 + k][e] - mu) * rs;
          if (gamma != nullptr) o[e] = fmaf(o[e], g[k][e], b[k][e]);
          o[e] = fb_act_apply_k<ACT>(act, o[e]);
        }
        if (c < d) st_piece<W>(yr + c, o);
      }
    }
  }
}

// Backward with dx.  A block's partial dgamma / dbeta: every thread's columns summed over its rows, then (T = 32) over the eight
// warps.  With the second kernel: 1001 features x 3000 rows 60 -> 42 us, 64 x 16384 58 -> 17, 3001 x 3000 163 -> 54, 8191 x 2000 331
// -> 114 (partials in global memory, rows read twice before).
template <int V, int T, bool VEC, int ACT>
__global__ void __launch_bounds__(LN_THREADS)
ln_bwd_rows_kernel(const float* __restrict__ x, const float* __restrict__ gamma, const float* __restrict__ beta,
                   const float* __restrict__ mean, const float* __restrict__ rstd, const float* __restrict__ dy, float* __restrict__ dx,
                   float* __restrict__ part_dg, float* __restrict__ part_db, int d, int64_t n, int act) {
  fb_after_previous();
  constexpr int W = VEC ? 4 : 1;
  __shared__ float sh[64];
  __shared__ float red[T == 32 ? 8 * V * W * 32 : 1];
  const int t = threadIdx.x % T, w = threadIdx.x / T;
  const float inv_d = 1.0f / (float)d;
  float ag[V][W], ab[V][W];
#pragma unroll
  for (int i = 0; i < V; ++i)
#pragma unroll
    for (int e = 0; e < W; ++e) ag[i][e] = ab[i][e] = 0.0f;
  for (int64_t row = (int64_t)blockIdx.x * (LN_THREADS / T) + w; row < n; row += (int64_t)gridDim.x * (LN_THREADS / T)) {
    const float mu = __ldg(mean + row), rs = __ldg(rstd + row);
    const float* xr = x + row * d;
    const float* dyr = dy + row * d;
    float xh[V][W], g[V][W];
#pragma unroll
    for (int i = 0; i < V; ++i) {
      const int c = (t + i * T) * W;
      if (c < d) {
        ld_piece<W>(xr + c, xh[i]);
        ld_piece<W>(dyr + c, g[i]);
      }
    }
    float s1 = 0.0f, s2 = 0.0f;
    float p[2][V];   // (of pieces of four)
#pragma unroll
    for (int i = 0; i < V; ++i) {
      const int c = (t + i * T) * W;
      p[0][i] = p[1][i] = 0.0f;
      if (c < d) {
        float ga[W], be[W];
        if (gamma != nullptr) {
          ld_piece<W>(gamma + c, ga);
          if (ACT != 0) ld_piece<W>(beta + c, be);
        }
#pragma unroll
        for (int e = 0; e < W; ++e) {
          if (gamma == nullptr) { ga[e] = 1.0f; be[e] = 0.0f; }
          const float h = (xh[i][e] - mu) * rs;
          const float dz = ACT == 0 ? g[i][e] : fb_act_bwd_k<ACT>(act, fmaf(h, ga[e], be[e]), g[i][e]);
          ag[i][e] = fmaf(dz, h, ag[i][e]);
          ab[i][e] += dz;
          xh[i][e] = h;
          g[i][e] = __fmul_rn(dz, ga[e]);
          if (!VEC) {
            s1 += g[i][e];
            s2 = fmaf(g[i][e], h, s2);
          }
        }
        if constexpr (VEC) {
          p[0][i] = sum4(g[i]);
          p[1][i] = dot4(g[i], xh[i]);
        }
      }
    }
    if constexpr (VEC) {
      float r[2];
      row_sums<V, 1, T>(p, r, sh);
      s1 = r[0]; s2 = r[1];
    } else if (T == 32) {
      s1 = fb_warp_sum(s1);
      s2 = fb_warp_sum(s2);
    } else {
      block_sum2(s1, s2, sh);
    }
    const float m1 = __fmul_rn(s1, inv_d), m2 = __fmul_rn(s2, inv_d);
    float* dxr = dx + row * d;
#pragma unroll
    for (int i = 0; i < V; ++i) {
      const int c = (t + i * T) * W;
      if (c < d) {
        float o[W];
#pragma unroll
        for (int e = 0; e < W; ++e) o[e] = rs * fmaf(-xh[i][e], m2, g[i][e] - m1);
        st_piece<W>(dxr + c, o);
      }
    }
  }
  if (part_dg == nullptr) return;
  float* pg = part_dg + (int64_t)blockIdx.x * d;
  float* pb = part_db + (int64_t)blockIdx.x * d;
  if (T != 32) {
#pragma unroll
    for (int i = 0; i < V; ++i) {
      const int c = (t + i * T) * W;
      if (c < d) {
        st_piece<W>(pg + c, ag[i]);
        st_piece<W>(pb + c, ab[i]);
      }
    }
    return;
  }
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    __syncthreads();
#pragma unroll
    for (int i = 0; i < V; ++i) st_piece<W>(red + w * (V * W * 32) + (t + i * 32) * W, k == 0 ? ag[i] : ab[i]);
    __syncthreads();
    for (int c = threadIdx.x; c < d; c += LN_THREADS) {
      float a = 0.0f;
#pragma unroll
      for (int r = 0; r < 8; ++r) a += red[r * (V * W * 32) + c];
      (k == 0 ? pg : pb)[c] = a;
    }
  }
}

// Only dgamma / dbeta: lx lanes side by side cover lx * W columns, 256 / lx rows at a time; grid (column blocks, row groups).
// dy counts dy_scale times.  Bound: one read of x and dy (1024 x 16384: 77 us with a dx, 38; 1001 x 3000: 60 and 17).
// CL: the row groups of a column block are a cluster, which adds its sums up itself (part_dg and part_db are dgamma and dbeta).
template <bool VEC, int ACT, bool CL, bool OWN>
__global__ void __launch_bounds__(LN_THREADS)
ln_bwd_params_kernel(const float* __restrict__ x, const float* __restrict__ gamma, const float* __restrict__ beta,
                     const float* __restrict__ mean, const float* __restrict__ rstd, const float* __restrict__ dy, float dy_scale,
                     float* __restrict__ part_dg, float* __restrict__ part_db, int64_t d, int64_t n, int act, int lx) {
  fb_after_previous();
  constexpr int W = VEC ? 4 : 1, U = 4;
  __shared__ float sa[LN_THREADS * W], sb[LN_THREADS * W];
  const int tx = threadIdx.x & (lx - 1), ty = threadIdx.x / lx, ny = LN_THREADS / lx;
  const int64_t c = ((int64_t)blockIdx.x * lx + tx) * W;
  float ag[W], ab[W], ga[W], be[W];
#pragma unroll
  for (int e = 0; e < W; ++e) { ag[e] = ab[e] = be[e] = 0.0f; ga[e] = 1.0f; }
  if (c < d) {
    if ((OWN || ACT != 0) && gamma != nullptr) {
      ld_piece<W>(gamma + c, ga);
      ld_piece<W>(beta + c, be);
    }
    const int64_t step = (int64_t)gridDim.y * ny;
    for (int64_t row = (int64_t)blockIdx.y * ny + ty; row < n; row += U * step) {
      float xv[U][W], dv[U][W], mu[U], rs[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int64_t r = row + u * step;
        const int64_t rr = r < n ? r : row;
        mu[u] = __ldg(mean + rr);
        rs[u] = __ldg(rstd + rr);
        ld_piece<W>(x + rr * d + c, xv[u]);
        if (!OWN) ld_piece<W>(dy + rr * d + c, dv[u]);
      }
#pragma unroll
      for (int u = 0; u < U; ++u)
#pragma unroll
        for (int e = 0; e < W; ++e) {
          if (row + u * step >= n) continue;
          const float h = (xv[u][e] - mu[u]) * rs[u];
          const float z = fmaf(h, ga[e], be[e]);
          float dz = (OWN ? fb_act_apply_k<ACT>(act, z) : dv[u][e]) * dy_scale;
          if (ACT != 0) dz = fb_act_bwd_k<ACT>(act, z, dz);
          ag[e] = fmaf(dz, h, ag[e]);
          ab[e] += dz;
        }
    }
  }
#pragma unroll
  for (int e = 0; e < W; ++e) { sa[threadIdx.x * W + e] = ag[e]; sb[threadIdx.x * W + e] = ab[e]; }
  __syncthreads();
  const int64_t col0 = (int64_t)blockIdx.x * lx * W;
  for (int k = threadIdx.x; k < lx * W; k += LN_THREADS) {
    if (!CL && col0 + k >= d) break;
    float a = 0.0f, b = 0.0f;
    for (int r = 0; r < ny; ++r) { a += sa[r * lx * W + k]; b += sb[r * lx * W + k]; }
    if (CL) {   // (column k's sums are this thread's: nobody else reads row 0 of it)
      sa[k] = a;
      sb[k] = b;
    } else {
      part_dg[(int64_t)blockIdx.y * d + col0 + k] = a;
      part_db[(int64_t)blockIdx.y * d + col0 + k] = b;
    }
  }
  if (CL) {
    cluster_column_sums(sa, lx * W, part_dg + col0, d - col0, gridDim.y);
    cluster_column_sums(sb, lx * W, part_db + col0, d - col0, gridDim.y);
  }
}

// ----------------------------------------------------------- BFloat16 arrays in and out ---
// The same sums, in the same order, on rows that are stored as BFloat16 (x, and dx with it; y and dy each by itself): between the
// layers of a bf16 model no Float32 copy of an array is made, and the results have the bits that such copies give.  Rows of up to 1024
// features belong to a warp, which reads eight values a lane at a time, rows of up to 8192 to a block, four a thread.  2048 rows of 4096: forward 44 us with its two casts, now 13; backward 48, now 18.
template <bool BF, int W>
struct Piece {
  static constexpr int N = BF ? W / 2 : W;   // words
  uint32_t w[N];
  __device__ __forceinline__ void load(const void* base, int64_t at) {
    const uint32_t* p = BF ? (const uint32_t*)((const uint16_t*)base + at) : (const uint32_t*)base + at;
    if constexpr (N == 2) {
      const uint2 a = *(const uint2*)p;
      w[0] = a.x; w[1] = a.y;
    } else {
#pragma unroll
      for (int i = 0; i < N; i += 4) {
        const uint4 a = *(const uint4*)(p + i);
        w[i] = a.x; w[i + 1] = a.y; w[i + 2] = a.z; w[i + 3] = a.w;
      }
    }
  }
  __device__ __forceinline__ void get(float (&v)[W]) const {
#pragma unroll
    for (int e = 0; e < W; ++e) v[e] = !BF ? __uint_as_float(w[e < N ? e : 0]) : __uint_as_float((e & 1) ? w[e / 2] & 0xffff0000u : w[e / 2] << 16);
  }
};
template <bool BF, int W>
__device__ __forceinline__ void put(void* base, int64_t at, const float (&v)[W]) {
  if constexpr (BF) {
    uint32_t b[W / 2];
#pragma unroll
    for (int e = 0; e < W / 2; ++e) b[e] = (uint32_t)fb_bf16_bits(v[2 * e]) | ((uint32_t)fb_bf16_bits(v[2 * e + 1]) << 16);
    if constexpr (W == 4) *(uint2*)((uint16_t*)base + at) = make_uint2(b[0], b[1]);
    else *(uint4*)((uint16_t*)base + at) = make_uint4(b[0], b[1], b[2], b[3]);
  } else {
#pragma unroll
    for (int e = 0; e < W; e += 4) *(float4*)((float*)base + at + e) = make_float4(v[e], v[e + 1], v[e + 2], v[e + 3]);
  }
}
template <int W>
__device__ __forceinline__ void ld_params(const float* p, float (&v)[W]) {
#pragma unroll
  for (int e = 0; e < W; e += 4) ld_piece<4>(p + e, v + e);
}

template <int V, int T, int ACT, bool XB, bool YB>
__global__ void __launch_bounds__(LN_THREADS)
ln_fwd_low_kernel(const void* __restrict__ x, const float* __restrict__ gamma, const float* __restrict__ beta, void* __restrict__ y,
                  float* __restrict__ mean, float* __restrict__ rstd, int d, int64_t n, float eps, int act) {
  fb_after_previous();
  constexpr int P = T == 32 ? 2 : 1, W = 4 * P;
  __shared__ float sh[64];
  const int t = threadIdx.x % T;
  const float inv_d = 1.0f / (float)d;
  for (int64_t row = (int64_t)blockIdx.x * (LN_THREADS / T) + threadIdx.x / T; row < n; row += (int64_t)gridDim.x * (LN_THREADS / T)) {
    float v[V][W];
    {
      Piece<XB, W> p[V];
#pragma unroll
      for (int i = 0; i < V; ++i)
        if ((t + i * T) * W < d) p[i].load(x, row * d + (t + i * T) * W);
#pragma unroll
      for (int i = 0; i < V; ++i) p[i].get(v[i]);
    }
    float mu, rs;
    row_stats<V, P, T>(v, t, d, inv_d, eps, sh, mu, rs);
    if (t == 0) {
      mean[row] = mu;
      rstd[row] = rs;
    }
#pragma unroll
    for (int i = 0; i < V; ++i) {
      const int c = (t + i * T) * W;
      if (c < d) {
        float g[W], b[W], o[W];
        if (gamma != nullptr) {
          ld_params(gamma + c, g);
          ld_params(beta + c, b);
        }
#pragma unroll
        for (int e = 0; e < W; ++e) {
          o[e] = (v[i][e] - mu) * rs;
          if (gamma != nullptr) o[e] = fmaf(o[e], g[e], b[e]);
          o[e] = fb_act_apply_k<ACT>(act, o[e]);
        }
        put<YB>(y, row * d + c, o);
      }
    }
  }
}

// dx has x's type; NULL leaves it out.  The next row's pieces are on their way while a row is summed.
template <int V, int T, int ACT, bool XB, bool DB>
__global__ void __launch_bounds__(LN_THREADS)
ln_bwd_low_kernel(const void* __restrict__ x, const float* __restrict__ gamma, const float* __restrict__ beta, const float* __restrict__ mean,
                  const float* __restrict__ rstd, const void* __restrict__ dy, void* __restrict__ dx, float* __restrict__ part_dg,
                  float* __restrict__ part_db, int d, int64_t n, int act) {
  fb_after_previous();
  constexpr int P = T == 32 ? 2 : 1, W = 4 * P;
  __shared__ float sh[64];
  __shared__ float red[T == 32 ? 8 * V * 32 * W : 1];
  const int t = threadIdx.x % T, w = threadIdx.x / T;
  const float inv_d = 1.0f / (float)d;
  float ag[V][W], ab[V][W];
#pragma unroll
  for (int i = 0; i < V; ++i)
#pragma unroll
    for (int e = 0; e < W; ++e) ag[i][e] = ab[i][e] = 0.0f;
  const int64_t step = (int64_t)gridDim.x * (LN_THREADS / T);
  int64_t row = (int64_t)blockIdx.x * (LN_THREADS / T) + w;
  Piece<XB, W> px[V];
  Piece<DB, W> pd[V];
  float mu1 = 0.0f, rs1 = 0.0f;
  auto fetch = [&](int64_t r) {
    if (r >= n) return;
    mu1 = __ldg(mean + r);
    rs1 = __ldg(rstd + r);
#pragma unroll
    for (int i = 0; i < V; ++i) {
      const int c = (t + i * T) * W;
      if (c < d) {
        px[i].load(x, r * d + c);
        pd[i].load(dy, r * d + c);
      }
    }
  };
  fetch(row);
  for (; row < n; row += step) {
    const float mu = mu1, rs = rs1;
    float xh[V][W], g[V][W];
#pragma unroll
    for (int i = 0; i < V; ++i) {
      px[i].get(xh[i]);
      pd[i].get(g[i]);
    }
    fetch(row + step);
    float p[2][V * P];
#pragma unroll
    for (int i = 0; i < V; ++i) {
      const int c = (t + i * T) * W;
#pragma unroll
      for (int h = 0; h < P; ++h) p[0][i * P + h] = p[1][i * P + h] = 0.0f;
      if (c < d) {
        float ga[W], be[W];
        if (gamma != nullptr) {
          ld_params(gamma + c, ga);
          if (ACT != 0) ld_params(beta + c, be);
        }
#pragma unroll
        for (int e = 0; e < W; ++e) {
          if (gamma == nullptr) { ga[e] = 1.0f; be[e] = 0.0f; }
          const float h = (xh[i][e] - mu) * rs;
          const float dz = ACT == 0 ? g[i][e] : fb_act_bwd_k<ACT>(act, fmaf(h, ga[e], be[e]), g[i][e]);
          ag[i][e] = fmaf(dz, h, ag[i][e]);
          ab[i][e] += dz;
          xh[i][e] = h;
          g[i][e] = __fmul_rn(dz, ga[e]);
        }
#pragma unroll
        for (int h = 0; h < P; ++h) {
          p[0][i * P + h] = sum4(g[i] + 4 * h);
          p[1][i * P + h] = dot4(g[i] + 4 * h, xh[i] + 4 * h);
        }
      }
    }
    if (dx == nullptr) continue;   // (uniform)
    float r[2];
    row_sums<V, P, T>(p, r, sh);
    const float m1 = __fmul_rn(r[0], inv_d), m2 = __fmul_rn(r[1], inv_d);
#pragma unroll
    for (int i = 0; i < V; ++i) {
      const int c = (t + i * T) * W;
      if (c < d) {
        float o[W];
#pragma unroll
        for (int e = 0; e < W; ++e) o[e] = rs * fmaf(-xh[i][e], m2, g[i][e] - m1);
        put<XB>(dx, row * d + c, o);
      }
    }
  }
  if (part_dg == nullptr) return;
  float* pg = part_dg + (int64_t)blockIdx.x * d;
  float* pb = part_db + (int64_t)blockIdx.x * d;
  if (T != 32) {
#pragma unroll
    for (int i = 0; i < V; ++i) {
      const int c = (t + i * T) * W;
      if (c < d) {
        put<false>(pg, c, ag[i]);
        put<false>(pb, c, ab[i]);
      }
    }
    return;
  }
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    __syncthreads();
#pragma unroll
    for (int i = 0; i < V; ++i) put<false>(red, w * (V * 32 * W) + (t + i * 32) * W, k == 0 ? ag[i] : ab[i]);
    __syncthreads();
    for (int c = threadIdx.x; c < d; c += LN_THREADS) {
      float a = 0.0f;
#pragma unroll
      for (int r = 0; r < 8; ++r) a += red[r * (V * 32 * W) + c];
      (k == 0 ? pg : pb)[c] = a;
    }
  }
}

// f(V, T) as compile-time constants for rows of d features
template <typename F>
void ln_low_dispatch(int64_t d, F f) {
  using std::integral_constant;
  if (d <= 256) f(integral_constant<int, 1>(), integral_constant<int, 32>());
  else if (d <= 512) f(integral_constant<int, 2>(), integral_constant<int, 32>());
  else if (d <= 1024) f(integral_constant<int, 4>(), integral_constant<int, 32>());
  else if (d <= 2048) f(integral_constant<int, 2>(), integral_constant<int, 256>());
  else if (d <= 4096) f(integral_constant<int, 4>(), integral_constant<int, 256>());
  else f(integral_constant<int, 8>(), integral_constant<int, 256>());
}
// f(first, second) of two flags as compile-time constants
template <typename F>
void ln_flags(bool a, bool b, F f) {
  if (a && b) f(std::true_type(), std::true_type());
  else if (a) f(std::true_type(), std::false_type());
  else if (b) f(std::false_type(), std::true_type());
  else f(std::false_type(), std::false_type());
}

// ------------------------------------------------------------------ forward, any d / alignment ---
__global__ void __launch_bounds__(LN_THREADS)
ln_fwd_generic_kernel(const float* __restrict__ x, const float* __restrict__ gamma,
                      const float* __restrict__ beta, float* __restrict__ y, float* __restrict__ mean,
                      float* __restrict__ rstd, int64_t d, int64_t n, float eps, int act) {
  fb_after_previous();
  __shared__ float sh[64];
  for (int64_t row = blockIdx.x; row < n; row += gridDim.x) {
    const float* xr = x + row * d;
    float s = 0.0f;
    for (int64_t c = threadIdx.x; c < d; c += LN_THREADS) s += xr[c];
    const float mu = fb_block_sum(s, sh) / (float)d;
    float q = 0.0f;
    for (int64_t c = threadIdx.x; c < d; c += LN_THREADS) { const float a = xr[c] - mu; q += a * a; }
    const float var = fb_block_sum(q, sh) / (float)d;
    const float rs = rsqrtf(var + eps);
    if (threadIdx.x == 0) { mean[row] = mu; rstd[row] = rs; }
    float* yr = y + row * d;
    for (int64_t c = threadIdx.x; c < d; c += LN_THREADS) {
      float o = (xr[c] - mu) * rs;
      if (gamma != nullptr) o = fmaf(o, gamma[c], beta[c]);
      yr[c] = fb_act_apply(act, o);
    }
  }
}

// ----------------------------------------------------------------- backward, row in registers ---
template <int V>
__global__ void __launch_bounds__(LN_THREADS, 2)
ln_bwd_vec_kernel(const float4* __restrict__ x, const float4* __restrict__ gamma,
                  const float4* __restrict__ beta, const float* __restrict__ mean,
                  const float* __restrict__ rstd, const float4* __restrict__ dy, float4* __restrict__ dx,
                  float4* __restrict__ part_dg, float4* __restrict__ part_db, int d4, int64_t n, int act) {
  fb_after_previous();
  __shared__ float sh[64];
  const float inv_d = 1.0f / (4.0f * (float)d4);
  float4 ag[V], ab[V], gam[V], bet[V];
#pragma unroll
  for (int i = 0; i < V; ++i) {
    const int c = threadIdx.x + i * LN_THREADS;
    ag[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    ab[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    gam[i] = (gamma != nullptr && c < d4) ? __ldg(gamma + c) : make_float4(1.f, 1.f, 1.f, 1.f);
    bet[i] = (beta != nullptr && c < d4) ? __ldg(beta + c) : make_float4(0.f, 0.f, 0.f, 0.f);
  }
  for (int64_t row = blockIdx.x; row < n; row += gridDim.x) {
    const float mu = __ldg(mean + row), rs = __ldg(rstd + row);
    const float4* xr = x + row * d4;
    const float4* dyr = dy + row * d4;
    float4 xh[V], g[V];
    float s1 = 0.0f, s2 = 0.0f;
#pragma unroll
    for (int i = 0; i < V; ++i) {
      const int c = threadIdx.x + i * LN_THREADS;
      if (c < d4) {
        const float4 xv = ld_stream(xr + c);
        float4 dz = ld_stream(dyr + c);
        xh[i].x = (xv.x - mu) * rs; xh[i].y = (xv.y - mu) * rs; xh[i].z = (xv.z - mu) * rs; xh[i].w = (xv.w - mu) * rs;
        if (act != FB_ACT_IDENTITY) {
          dz.x *= fb_act_grad_z(act, fmaf(xh[i].x, gam[i].x, bet[i].x));
          dz.y *= fb_act_grad_z(act, fmaf(xh[i].y, gam[i].y, bet[i].y));
          dz.z *= fb_act_grad_z(act, fmaf(xh[i].z, gam[i].z, bet[i].z));
          dz.w *= fb_act_grad_z(act, fmaf(xh[i].w, gam[i].w, bet[i].w));
        }
        ag[i].x = fmaf(dz.x, xh[i].x, ag[i].x); ag[i].y = fmaf(dz.y, xh[i].y, ag[i].y);
        ag[i].z = fmaf(dz.z, xh[i].z, ag[i].z); ag[i].w = fmaf(dz.w, xh[i].w, ag[i].w);
        ab[i].x += dz.x; ab[i].y += dz.y; ab[i].z += dz.z; ab[i].w += dz.w;
        g[i].x = dz.x * gam[i].x; g[i].y = dz.y * gam[i].y; g[i].z = dz.z * gam[i].z; g[i].w = dz.w * gam[i].w;
        s1 += (g[i].x + g[i].y) + (g[i].z + g[i].w);
        s2 += (g[i].x * xh[i].x + g[i].y * xh[i].y) + (g[i].z * xh[i].z + g[i].w * xh[i].w);
      }
    }
    block_sum2(s1, s2, sh);
    const float m1 = __fmul_rn(s1, inv_d), m2 = __fmul_rn(s2, inv_d);
    float4* dxr = dx + row * d4;
#pragma unroll
    for (int i = 0; i < V; ++i) {
      const int c = threadIdx.x + i * LN_THREADS;
      if (c < d4) {
        float4 o;
        o.x = rs * (g[i].x - m1 - xh[i].x * m2); o.y = rs * (g[i].y - m1 - xh[i].y * m2);
        o.z = rs * (g[i].z - m1 - xh[i].z * m2); o.w = rs * (g[i].w - m1 - xh[i].w * m2);
        st_stream(dxr + c, o);
      }
    }
  }
  if (part_dg != nullptr) {
#pragma unroll
    for (int i = 0; i < V; ++i) {
      const int c = threadIdx.x + i * LN_THREADS;
      if (c < d4) {
        part_dg[(int64_t)blockIdx.x * d4 + c] = ag[i];
        part_db[(int64_t)blockIdx.x * d4 + c] = ab[i];
      }
    }
  }
}

// ------------------------------------------- backward, rows staged through shared memory ---
// Same arithmetic as ln_bwd_vec_kernel, but the x and dy rows of the next LN_PIPE - 1 iterations are already in
// flight (cp.async.bulk into a ring of shared-memory stages) while the current row is reduced, so the kernel does
// not depend on occupancy for memory-level parallelism.
constexpr int LN_PIPE_MAX = 3;
constexpr size_t LN_PIPE_BYTES = 100 * 1024;   // of all stages
constexpr uint32_t LN_WAIT_LIMIT = 1u << 22;

__device__ __forceinline__ uint32_t ln_smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

template <int V>
__global__ void __launch_bounds__(LN_THREADS, 2)
ln_bwd_pipe_kernel(const float* __restrict__ x, const float4* __restrict__ gamma, const float4* __restrict__ beta,
                   const float* __restrict__ mean, const float* __restrict__ rstd, const float* __restrict__ dy,
                   float4* __restrict__ dx, float4* __restrict__ part_dg, float4* __restrict__ part_db, int d4,
                   int64_t n, int act, int nstages, int32_t* __restrict__ dev_err) {
  fb_after_previous();
  extern __shared__ __align__(128) uint8_t ln_smem[];
  __shared__ float sh[64];
  __shared__ __align__(8) uint64_t bar[LN_PIPE_MAX];
  __shared__ int s_fail;
  const uint32_t row_bytes = (uint32_t)d4 * 16u;
  float4* stage_base = (float4*)ln_smem;                 // stage s: x row at [s][0], dy row at [s][1]
  const float inv_d = 1.0f / (4.0f * (float)d4);
  const int64_t first = blockIdx.x, step = gridDim.x;
  const int64_t my_rows = first < n ? (n - first + step - 1) / step : 0;

  auto issue = [&](int64_t i) {   // one thread: bring row first + i*step into stage i % nstages
    const int s = (int)(i % nstages);
    const int64_t row = first + i * step;
    const uint32_t b = ln_smem_u32(&bar[s]);
    const uint32_t dst_x = ln_smem_u32(stage_base + (size_t)(2 * s) * d4);
    const uint32_t dst_d = ln_smem_u32(stage_base + (size_t)(2 * s + 1) * d4);
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(b), "r"(2u * row_bytes) : "memory");
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(dst_x), "l"(x + row * (int64_t)d4 * 4), "r"(row_bytes), "r"(b) : "memory");
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(dst_d), "l"(dy + row * (int64_t)d4 * 4), "r"(row_bytes), "r"(b) : "memory");
  };

  if (threadIdx.x == 0) {
    for (int s = 0; s < nstages; ++s)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(ln_smem_u32(&bar[s])) : "memory");
    s_fail = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    for (int64_t i = 0; i < nstages && i < my_rows; ++i) issue(i);
  }
  __syncthreads();

  float4 ag[V], ab[V], gam[V], bet[V];
#pragma unroll
  for (int i = 0; i < V; ++i) {
    const int c = threadIdx.x + i * LN_THREADS;
    ag[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    ab[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    gam[i] = (gamma != nullptr && c < d4) ? __ldg(gamma + c) : make_float4(1.f, 1.f, 1.f, 1.f);
    bet[i] = (beta != nullptr && c < d4) ? __ldg(beta + c) : make_float4(0.f, 0.f, 0.f, 0.f);
  }
  for (int64_t it = 0; it < my_rows; ++it) {
    const int s = (int)(it % nstages);
    const uint32_t parity = (uint32_t)(it / nstages) & 1u;
    const int64_t row = first + it * step;
    {
      // bounded wait for this stage's two bulk copies
      const uint32_t b = ln_smem_u32(&bar[s]);
      uint32_t ok = 0;
      for (uint32_t spin = 0; spin < LN_WAIT_LIMIT && !ok; ++spin)
        asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                     : "=r"(ok) : "r"(b), "r"(parity) : "memory");
      if (!ok) s_fail = 1;
    }
    const float mu = __ldg(mean + row), rs = __ldg(rstd + row);
    const float4* xr = stage_base + (size_t)(2 * s) * d4;
    const float4* dyr = stage_base + (size_t)(2 * s + 1) * d4;
    float4 xh[V], g[V];
    float s1 = 0.0f, s2 = 0.0f;
#pragma unroll
    for (int i = 0; i < V; ++i) {
      const int c = threadIdx.x + i * LN_THREADS;
      if (c < d4) {
        const float4 xv = xr[c];
        float4 dz = dyr[c];
        xh[i].x = (xv.x - mu) * rs; xh[i].y = (xv.y - mu) * rs; xh[i].z = (xv.z - mu) * rs; xh[i].w = (xv.w - mu) * rs;
        if (act != FB_ACT_IDENTITY) {
          dz.x *= fb_act_grad_z(act, fmaf(xh[i].x, gam[i].x, bet[i].x));
          dz.y *= fb_act_grad_z(act, fmaf(xh[i].y, gam[i].y, bet[i].y));
          dz.z *= fb_act_grad_z(act, fmaf(xh[i].z, gam[i].z, bet[i].z));
          dz.w *= fb_act_grad_z(act, fmaf(xh[i].w, gam[i].w, bet[i].w));
        }
        ag[i].x = fmaf(dz.x, xh[i].x, ag[i].x); ag[i].y = fmaf(dz.y, xh[i].y, ag[i].y);
        ag[i].z = fmaf(dz.z, xh[i].z, ag[i].z); ag[i].w = fmaf(dz.w, xh[i].w, ag[i].w);
        ab[i].x += dz.x; ab[i].y += dz.y; ab[i].z += dz.z; ab[i].w += dz.w;
        g[i].x = dz.x * gam[i].x; g[i].y = dz.y * gam[i].y; g[i].z = dz.z * gam[i].z; g[i].w = dz.w * gam[i].w;
        s1 += (g[i].x + g[i].y) + (g[i].z + g[i].w);
        s2 += (g[i].x * xh[i].x + g[i].y * xh[i].y) + (g[i].z * xh[i].z + g[i].w * xh[i].w);
      }
    }
    block_sum2(s1, s2, sh);   // its barriers also mean: every thread has finished reading stage s
    if (s_fail) break;        // block-uniform after the barriers above
    if (threadIdx.x == 0 && it + nstages < my_rows) issue(it + nstages);
    const float m1 = __fmul_rn(s1, inv_d), m2 = __fmul_rn(s2, inv_d);
    float4* dxr = dx + row * d4;
#pragma unroll
    for (int i = 0; i < V; ++i) {
      const int c = threadIdx.x + i * LN_THREADS;
      if (c < d4) {
        float4 o;
        o.x = rs * (g[i].x - m1 - xh[i].x * m2); o.y = rs * (g[i].y - m1 - xh[i].y * m2);
        o.z = rs * (g[i].z - m1 - xh[i].z * m2); o.w = rs * (g[i].w - m1 - xh[i].w * m2);
        st_stream(dxr + c, o);
      }
    }
  }
  if (part_dg != nullptr) {
#pragma unroll
    for (int i = 0; i < V; ++i) {
      const int c = threadIdx.x + i * LN_THREADS;
      if (c < d4) {
        part_dg[(int64_t)blockIdx.x * d4 + c] = ag[i];
        part_db[(int64_t)blockIdx.x * d4 + c] = ab[i];
      }
    }
  }
  if (threadIdx.x == 0 && s_fail && dev_err != nullptr) atomicExch(dev_err, 2001);
}

// ---------------------------------------------------------------- backward, any d / alignment ---
__global__ void __launch_bounds__(LN_THREADS)
ln_bwd_generic_kernel(const float* __restrict__ x, const float* __restrict__ gamma,
                      const float* __restrict__ beta, const float* __restrict__ mean,
                      const float* __restrict__ rstd, const float* __restrict__ dy, float* __restrict__ dx,
                      float* __restrict__ part_dg, float* __restrict__ part_db, int64_t d, int64_t n, int act) {
  fb_after_previous();
  __shared__ float sh[64];
  float* pg = part_dg ? part_dg + (int64_t)blockIdx.x * d : nullptr;
  float* pb = part_db ? part_db + (int64_t)blockIdx.x * d : nullptr;
  if (pg)
    for (int64_t c = threadIdx.x; c < d; c += LN_THREADS) { pg[c] = 0.0f; pb[c] = 0.0f; }
  for (int64_t row = blockIdx.x; row < n; row += gridDim.x) {
    const float mu = mean[row], rs = rstd[row];
    const float* xr = x + row * d;
    const float* dyr = dy + row * d;
    float s1 = 0.0f, s2 = 0.0f;
    for (int64_t c = threadIdx.x; c < d; c += LN_THREADS) {
      const float xh = (xr[c] - mu) * rs;
      const float ga = gamma ? gamma[c] : 1.0f, be = beta ? beta[c] : 0.0f;
      const float dz = dyr[c] * fb_act_grad_z(act, fmaf(xh, ga, be));
      const float g = dz * ga;
      s1 += g;
      s2 += g * xh;
    }
    block_sum2(s1, s2, sh);
    const float m1 = s1 / (float)d, m2 = s2 / (float)d;
    float* dxr = dx + row * d;
    for (int64_t c = threadIdx.x; c < d; c += LN_THREADS) {
      const float xh = (xr[c] - mu) * rs;
      const float ga = gamma ? gamma[c] : 1.0f, be = beta ? beta[c] : 0.0f;
      const float dz = dyr[c] * fb_act_grad_z(act, fmaf(xh, ga, be));
      dxr[c] = rs * (dz * ga - m1 - xh * m2);
      if (pg) { pg[c] += dz * xh; pb[c] += dz; }   // column c is always owned by this thread
    }
  }
}

}  // namespace

// out_a[j] = sum_g part_a[g][j], out_b[j] = sum_g part_b[g][j]; block = 32 columns x 8 row groups.
__global__ void __launch_bounds__(256)
fb_colreduce2_kernel(const float* __restrict__ part_a, const float* __restrict__ part_b,
                     float* __restrict__ out_a, float* __restrict__ out_b, int64_t groups, int64_t d) {
  fb_after_previous();
  fb_let_next_start();
  __shared__ float sa[8][33], sb[8][33];
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const int64_t col = (int64_t)blockIdx.x * 32 + tx;
  float a = 0.0f, b = 0.0f;
  if (col < d) {
    // four independent loads per array in flight
    int64_t g = ty;
    for (; g + 24 < groups; g += 32) {
      const float a0 = part_a[g * d + col], a1 = part_a[(g + 8) * d + col], a2 = part_a[(g + 16) * d + col], a3 = part_a[(g + 24) * d + col];
      float b0 = 0.f, b1 = 0.f, b2 = 0.f, b3 = 0.f;
      if (part_b) { b0 = part_b[g * d + col]; b1 = part_b[(g + 8) * d + col]; b2 = part_b[(g + 16) * d + col]; b3 = part_b[(g + 24) * d + col]; }
      a += (a0 + a1) + (a2 + a3);
      b += (b0 + b1) + (b2 + b3);
    }
    for (; g < groups; g += 8) {
      a += part_a[g * d + col];
      if (part_b) b += part_b[g * d + col];
    }
  }
  sa[ty][tx] = a;
  sb[ty][tx] = b;
  __syncthreads();
  if (ty == 0 && col < d) {
#pragma unroll
    for (int i = 1; i < 8; ++i) { a += sa[i][tx]; b += sb[i][tx]; }
    out_a[col] = a;
    if (out_b) out_b[col] = b;
  }
}

// f(V, T, VEC) as compile-time constants for the kernels that hold rows of d features in registers; false: none does.  Aligned
// rows of more than 1024 features keep the kernels above, whose rows stream past L2.
template <typename F>
static bool ln_rows_dispatch(int64_t d, bool vec, F f) {
  using std::integral_constant;
  using std::true_type;
  using std::false_type;
  if (vec) {
    if (d <= 128) f(integral_constant<int, 1>(), integral_constant<int, 32>(), true_type());
    else if (d <= 256) f(integral_constant<int, 2>(), integral_constant<int, 32>(), true_type());
    else if (d <= 512) f(integral_constant<int, 4>(), integral_constant<int, 32>(), true_type());
    else if (d <= 1024) f(integral_constant<int, 8>(), integral_constant<int, 32>(), true_type());
    else return false;
    return true;
  }
  if (d <= 128) f(integral_constant<int, 4>(), integral_constant<int, 32>(), false_type());
  else if (d <= 256) f(integral_constant<int, 8>(), integral_constant<int, 32>(), false_type());
  else if (d <= 512) f(integral_constant<int, 16>(), integral_constant<int, 32>(), false_type());
  else if (d <= 1024) f(integral_constant<int, 32>(), integral_constant<int, 32>(), false_type());
  else if (d <= 2048) f(integral_constant<int, 8>(), integral_constant<int, 256>(), false_type());
  else if (d <= 4096) f(integral_constant<int, 16>(), integral_constant<int, 256>(), false_type());
  else if (d <= 8192) f(integral_constant<int, 32>(), integral_constant<int, 256>(), false_type());
  else return false;
  return true;
}

static int ln_pick_v(int64_t d4) {
  const int64_t per = (d4 + LN_THREADS - 1) / LN_THREADS;
  if (per <= 2) return 2;
  if (per <= 4) return 4;
  if (per <= 8) return 8;
  return 0;
}

FB_API int32_t fb_layernorm_fwd(fb_ctx* ctx, void* stream_, const float* x, const float* gamma,
                                const float* beta, float* y, float* mean, float* rstd, int64_t d, int64_t n,
                                float eps, int32_t act) {
  FB_CHECK_CTX(ctx);
  cudaStream_t stream = (cudaStream_t)stream_;
  FB_REQUIRE(d >= 1 && n >= 0, FB_ERR_SHAPE, "fb_layernorm_fwd: bad shape d=%lld n=%lld", (long long)d, (long long)n);
  FB_REQUIRE(fb_act_valid(act), FB_ERR_INVALID_ARG, "fb_layernorm_fwd: unknown activation %d", act);
  FB_REQUIRE((gamma == nullptr) == (beta == nullptr), FB_ERR_INVALID_ARG, "fb_layernorm_fwd: gamma and beta must both be given or both NULL");
  if (n == 0) return FB_OK;
  FB_REQUIRE(x && y && mean && rstd, FB_ERR_INVALID_ARG, "fb_layernorm_fwd: NULL pointer");
  const bool vec = (d % 4 == 0) && fb_aligned16(x) && fb_aligned16(y) && (!gamma || (fb_aligned16(gamma) && fb_aligned16(beta)));
  const int v = vec ? ln_pick_v(d / 4) : 0;
  const unsigned grid = (unsigned)(n < (int64_t)ctx->sm_count * 64 ? n : (int64_t)ctx->sm_count * 64);
  const bool rows = ln_rows_dispatch(d, vec, [&](auto V, auto T, auto vc) {
    const int64_t per = LN_THREADS / T.value, blocks = (n + per - 1) / per;
    fb_act_kind(act, [&](auto k) {
      fb_launch(ln_fwd_rows_kernel<V.value, T.value, vc.value, k.value>, (unsigned)(blocks < 0x7fffffff ? blocks : 0x7fffffff), LN_THREADS, 0, stream, x, gamma, beta, y, mean, rstd, (int)d, n, eps, act);
    });
  });
  if (rows) {
  } else if (v == 0) {
    fb_launch(ln_fwd_generic_kernel, grid, LN_THREADS, 0, stream, x, gamma, beta, y, mean, rstd, d, n, eps, act);
  } else {
    const float4 *x4 = (const float4*)x, *g4 = (const float4*)gamma, *b4 = (const float4*)beta;
    float4* y4 = (float4*)y;
    const int d4 = (int)(d / 4);
    const unsigned gridv = (unsigned)(n < 0x7fffffff ? n : 0x7fffffff);
    switch (v) {
      case 2: fb_launch(ln_fwd_vec_kernel<2>, gridv, LN_THREADS, 0, stream, x4, g4, b4, y4, mean, rstd, d4, n, eps, act); break;
      case 4: fb_launch(ln_fwd_vec_kernel<4>, gridv, LN_THREADS, 0, stream, x4, g4, b4, y4, mean, rstd, d4, n, eps, act); break;
      default: fb_launch(ln_fwd_vec_kernel<8>, gridv, LN_THREADS, 0, stream, x4, g4, b4, y4, mean, rstd, d4, n, eps, act); break;
    }
  }
  FB_LAUNCH_CHECK();
  return FB_OK;
}

// Launches the backward kernels; `part` holds 2 * groups * d floats of per-block partials.
int32_t fb_layernorm_bwd_impl(cudaStream_t stream, int sm_count, float* part, int64_t groups, const float* x,
                              const float* gamma, const float* beta, const float* mean, const float* rstd,
                              const float* dy, float* dx, float* dgamma, float* dbeta, int64_t d, int64_t n,
                              int32_t act, int32_t* dev_err, bool allow_ring = true) {
  (void)sm_count;
  if (d <= 1024 && groups > (n + 7) / 8) groups = (n + 7) / 8;   // (eight rows a block)
  const bool want_param = (dgamma != nullptr);
  float* part_dg = want_param ? part : nullptr;
  float* part_db = want_param ? part + groups * d : nullptr;
  const bool vec = (d % 4 == 0) && fb_aligned16(x) && fb_aligned16(dy) && fb_aligned16(dx) &&
                   (!gamma || (fb_aligned16(gamma) && fb_aligned16(beta)));
  const int v = vec ? ln_pick_v(d / 4) : 0;
  const bool rows = ln_rows_dispatch(d, vec, [&](auto V, auto T, auto vc) {
    fb_act_kind(act, [&](auto k) {
      fb_launch(ln_bwd_rows_kernel<V.value, T.value, vc.value, k.value>, (unsigned)groups, LN_THREADS, 0, stream, x, gamma, beta, mean, rstd, dy, dx, part_dg, part_db, (int)d, n, act);
    });
  });
  if (rows) {
  } else if (v == 0) {
    fb_launch(ln_bwd_generic_kernel, (unsigned)groups, LN_THREADS, 0, stream, x, gamma, beta, mean, rstd, dy, dx, part_dg,
                                                                       part_db, d, n, act);
  } else {
    const float4 *x4 = (const float4*)x, *g4 = (const float4*)gamma, *b4 = (const float4*)beta, *dy4 = (const float4*)dy;
    float4 *dx4 = (float4*)dx, *pg4 = (float4*)part_dg, *pb4 = (float4*)part_db;
    const int d4 = (int)(d / 4);
    const unsigned g = (unsigned)groups;
    // rows staged through shared memory when at least two stages of (x row, dy row) fit beside a second block
    const size_t stage_bytes = (size_t)2 * d * sizeof(float);
    int nst = (int)(LN_PIPE_BYTES / stage_bytes);
    if (nst > LN_PIPE_MAX) nst = LN_PIPE_MAX;
    if (nst >= 2 && v >= 2 && allow_ring) {
      const size_t smem = (size_t)nst * stage_bytes;
      switch (v) {
        case 2:
          FB_CUDA(fb_allow_smem(ln_bwd_pipe_kernel<2>, LN_PIPE_BYTES));
          fb_launch(ln_bwd_pipe_kernel<2>, g, LN_THREADS, smem, stream, x, g4, b4, mean, rstd, dy, dx4, pg4, pb4, d4, n, act, nst, dev_err);
          break;
        case 4:
          FB_CUDA(fb_allow_smem(ln_bwd_pipe_kernel<4>, LN_PIPE_BYTES));
          fb_launch(ln_bwd_pipe_kernel<4>, g, LN_THREADS, smem, stream, x, g4, b4, mean, rstd, dy, dx4, pg4, pb4, d4, n, act, nst, dev_err);
          break;
        default:
          FB_CUDA(fb_allow_smem(ln_bwd_pipe_kernel<8>, LN_PIPE_BYTES));
          fb_launch(ln_bwd_pipe_kernel<8>, g, LN_THREADS, smem, stream, x, g4, b4, mean, rstd, dy, dx4, pg4, pb4, d4, n, act, nst, dev_err);
          break;
      }
    } else {
      switch (v) {
        case 2: fb_launch(ln_bwd_vec_kernel<2>, g, LN_THREADS, 0, stream, x4, g4, b4, mean, rstd, dy4, dx4, pg4, pb4, d4, n, act); break;
        case 4: fb_launch(ln_bwd_vec_kernel<4>, g, LN_THREADS, 0, stream, x4, g4, b4, mean, rstd, dy4, dx4, pg4, pb4, d4, n, act); break;
        default: fb_launch(ln_bwd_vec_kernel<8>, g, LN_THREADS, 0, stream, x4, g4, b4, mean, rstd, dy4, dx4, pg4, pb4, d4, n, act); break;
      }
    }
  }
  FB_LAUNCH_CHECK();
  if (want_param) {
    fb_launch(fb_colreduce2_kernel, (unsigned)((d + 31) / 32), 256, 0, stream, part_dg, part_db, dgamma, dbeta, groups, d);
    FB_LAUNCH_CHECK();
  }
  return FB_OK;
}

int64_t fb_layernorm_bwd_groups(int sm_count, int64_t n) {
  int64_t groups = (int64_t)sm_count * 2;
  if (groups > n) groups = n;
  if (groups < 1) groups = 1;
  return groups;
}

FB_API int32_t fb_layernorm_bwd(fb_ctx* ctx, void* stream_, const float* x, const float* gamma,
                                const float* beta, const float* mean, const float* rstd, const float* dy,
                                float* dx, float* dgamma, float* dbeta, int64_t d, int64_t n, int32_t act) {
  FB_CHECK_CTX(ctx);
  cudaStream_t stream = (cudaStream_t)stream_;
  FB_REQUIRE(d >= 1 && n >= 0, FB_ERR_SHAPE, "fb_layernorm_bwd: bad shape d=%lld n=%lld", (long long)d, (long long)n);
  FB_REQUIRE(fb_act_valid(act), FB_ERR_INVALID_ARG, "fb_layernorm_bwd: unknown activation %d", act);
  FB_REQUIRE((gamma == nullptr) == (beta == nullptr), FB_ERR_INVALID_ARG, "fb_layernorm_bwd: gamma and beta must both be given or both NULL");
  FB_REQUIRE((dgamma == nullptr) == (dbeta == nullptr), FB_ERR_INVALID_ARG, "fb_layernorm_bwd: dgamma and dbeta must both be given or both NULL");
  if (n == 0) {
    if (dgamma) {
      FB_CUDA(cudaMemsetAsync(dgamma, 0, d * sizeof(float), stream));
      FB_CUDA(cudaMemsetAsync(dbeta, 0, d * sizeof(float), stream));
    }
    return FB_OK;
  }
  FB_REQUIRE(x && mean && rstd && dy && dx, FB_ERR_INVALID_ARG, "fb_layernorm_bwd: NULL pointer");
  const int64_t groups = fb_layernorm_bwd_groups(ctx->sm_count, n);
  float* part = nullptr;
  if (dgamma) {
    part = (float*)fb_scratch(ctx, stream, (size_t)(2 * groups * d) * sizeof(float));
    if (!part) return FB_ERR_ALLOC;
  }
  return fb_layernorm_bwd_impl(stream, ctx->sm_count, part, groups, x, gamma, beta, mean, rstd, dy, dx, dgamma, dbeta,
                               d, n, act, ctx->dev_error);
}

// dy == NULL: the cotangent is dy_scale times the layer's output, which the kernel makes from x instead of reading it
static int32_t ln_bwd_params(const char* fn, fb_ctx* ctx, cudaStream_t stream, const float* x, const float* gamma, const float* beta,
                             const float* mean, const float* rstd, const float* dy, float dy_scale, float* dgamma,
                             float* dbeta, int64_t d, int64_t n, int32_t act) {
  FB_REQUIRE(d >= 1 && n >= 0, FB_ERR_SHAPE, "%s: bad shape d=%lld n=%lld", fn, (long long)d, (long long)n);
  FB_REQUIRE(fb_act_valid(act), FB_ERR_INVALID_ARG, "%s: unknown activation %d", fn, act);
  FB_REQUIRE((gamma == nullptr) == (beta == nullptr), FB_ERR_INVALID_ARG, "%s: gamma and beta must both be given or both NULL", fn);
  FB_REQUIRE(dgamma && dbeta, FB_ERR_INVALID_ARG, "%s: NULL pointer", fn);
  if (n == 0) {
    FB_CUDA(cudaMemsetAsync(dgamma, 0, d * sizeof(float), stream));
    FB_CUDA(cudaMemsetAsync(dbeta, 0, d * sizeof(float), stream));
    return FB_OK;
  }
  FB_REQUIRE(x && mean && rstd, FB_ERR_INVALID_ARG, "%s: NULL pointer", fn);
  const bool vec = (d % 4 == 0) && fb_aligned16(x) && (dy == nullptr || fb_aligned16(dy)) && (!gamma || (fb_aligned16(gamma) && fb_aligned16(beta)));
  const int64_t pieces = vec ? d / 4 : d;
  int lx = 32;
  while (lx > 1 && lx / 2 >= pieces) lx /= 2;
  // about eight blocks per SM, each with at least four rows a thread
  const int64_t col_blocks = (pieces + lx - 1) / lx, ny = LN_THREADS / lx;
  // Where eight row groups leave a thread no more than 8 rows they are one cluster, without a second kernel (with 47 rows a thread,
  // 1001 x 3000, that takes 20.1 us against 10.8 and 4.2).
  const bool one = n <= 8 * 8 * ny && col_blocks <= 0xfffffff;
  int64_t groups = one ? 8 : ((int64_t)ctx->sm_count * 8 + col_blocks - 1) / col_blocks;
  const int64_t most = (n + 4 * ny - 1) / (4 * ny);
  groups = groups > most ? most : groups;
  groups = groups > 65535 ? 65535 : groups;
  FB_REQUIRE(col_blocks <= 0x7fffffff, FB_ERR_UNSUPPORTED, "%s: too many features", fn);
  if (one) {
    cudaLaunchConfig_t lc;
    memset(&lc, 0, sizeof(lc));
    lc.gridDim = dim3((unsigned)col_blocks, (unsigned)groups, 1);
    lc.blockDim = dim3(LN_THREADS, 1, 1);
    lc.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = attr[0].val.clusterDim.z = 1;
    attr[0].val.clusterDim.y = (unsigned)groups;
    lc.attrs = attr;
    lc.numAttrs = 1;
    const cudaError_t e = fb_act_kind(act, [&](auto k) {
      return cudaLaunchKernelEx(&lc, dy == nullptr ? (vec ? ln_bwd_params_kernel<true, k.value, true, true> : ln_bwd_params_kernel<false, k.value, true, true>)
                                                   : (vec ? ln_bwd_params_kernel<true, k.value, true, false> : ln_bwd_params_kernel<false, k.value, true, false>),
                                x, gamma, beta, mean, rstd, dy, dy_scale, dgamma, dbeta, d, n, (int)act, lx);
    });
    FB_CUDA(e);
    FB_LAUNCH_CHECK();
    return FB_OK;
  }
  float* part = (float*)fb_scratch(ctx, stream, (size_t)(2 * groups * d) * sizeof(float));
  if (!part) return FB_ERR_ALLOC;
  float *pg = part, *pb = part + groups * d;
  const dim3 grid((unsigned)col_blocks, (unsigned)groups);
  fb_act_kind(act, [&](auto k) {
    auto kern = dy == nullptr ? (vec ? ln_bwd_params_kernel<true, k.value, false, true> : ln_bwd_params_kernel<false, k.value, false, true>)
                              : (vec ? ln_bwd_params_kernel<true, k.value, false, false> : ln_bwd_params_kernel<false, k.value, false, false>);
    fb_launch(kern, grid, LN_THREADS, 0, stream, x, gamma, beta, mean, rstd, dy, dy_scale, pg, pb, d, n, act, lx);
  });
  FB_LAUNCH_CHECK();
  fb_launch(fb_colreduce2_kernel, (unsigned)((d + 31) / 32), 256, 0, stream, pg, pb, dgamma, dbeta, groups, d);
  FB_LAUNCH_CHECK();
  return FB_OK;
}

FB_API int32_t fb_layernorm_bwd_params(fb_ctx* ctx, void* stream, const float* x, const float* gamma, const float* beta,
                                       const float* mean, const float* rstd, const float* dy, float dy_scale, float* dgamma,
                                       float* dbeta, int64_t d, int64_t n, int32_t act) {
  FB_CHECK_CTX(ctx);
  FB_REQUIRE(dy != nullptr || n <= 0, FB_ERR_INVALID_ARG, "fb_layernorm_bwd_params: NULL pointer");
  return ln_bwd_params("fb_layernorm_bwd_params", ctx, (cudaStream_t)stream, x, gamma, beta, mean, rstd, dy, dy_scale, dgamma, dbeta, d, n, act);
}

FB_API int32_t fb_layernorm_bwd_params_own(fb_ctx* ctx, void* stream, const float* x, const float* gamma, const float* beta,
                                           const float* mean, const float* rstd, float y_scale, float* dgamma, float* dbeta, int64_t d,
                                           int64_t n, int32_t act) {
  FB_CHECK_CTX(ctx);
  return ln_bwd_params("fb_layernorm_bwd_params_own", ctx, (cudaStream_t)stream, x, gamma, beta, mean, rstd, nullptr, y_scale, dgamma, dbeta, d, n, act);
}

static bool ln_low_ok(const void* x, const float* gamma, const float* beta, const void* b, const void* c, int64_t d) {
  return d % 8 == 0 && d <= 8192 && fb_aligned16(x) && fb_aligned16(b) && fb_aligned16(c) && fb_aligned16(gamma) && fb_aligned16(beta);
}

FB_API int32_t fb_layernorm_fwd_mixed(fb_ctx* ctx, void* stream_, const void* x, int32_t x_bf16, const float* gamma, const float* beta, void* y,
                                      int32_t y_bf16, float* mean, float* rstd, int64_t d, int64_t n, float eps, int32_t act) {
  FB_CHECK_CTX(ctx);
  cudaStream_t stream = (cudaStream_t)stream_;
  FB_REQUIRE(d >= 1 && n >= 0, FB_ERR_SHAPE, "fb_layernorm_fwd_mixed: bad shape d=%lld n=%lld", (long long)d, (long long)n);
  FB_REQUIRE(fb_act_valid(act), FB_ERR_INVALID_ARG, "fb_layernorm_fwd_mixed: unknown activation %d", act);
  FB_REQUIRE((gamma == nullptr) == (beta == nullptr), FB_ERR_INVALID_ARG, "fb_layernorm_fwd_mixed: gamma and beta must both be given or both NULL");
  if (n == 0) return FB_OK;
  FB_REQUIRE(x && y && mean && rstd, FB_ERR_INVALID_ARG, "fb_layernorm_fwd_mixed: NULL pointer");
  FB_REQUIRE(ln_low_ok(x, gamma, beta, y, nullptr, d), FB_ERR_UNSUPPORTED, "fb_layernorm_fwd_mixed: needs 16-byte aligned arrays and a multiple of 8 up to 8192 features");
  ln_low_dispatch(d, [&](auto V, auto T) {
    const int64_t per = LN_THREADS / T.value, blocks = (n + per - 1) / per;
    const unsigned grid = (unsigned)(blocks < 0x7fffffff ? blocks : 0x7fffffff);
    fb_act_kind(act, [&](auto k) {
      ln_flags(x_bf16 != 0, y_bf16 != 0, [&](auto xb, auto yb) {
        fb_launch(ln_fwd_low_kernel<V.value, T.value, k.value, xb.value, yb.value>, grid, LN_THREADS, 0, stream, x, gamma, beta, y, mean, rstd, (int)d, n, eps, act);
      });
    });
  });
  FB_LAUNCH_CHECK();
  return FB_OK;
}

FB_API int32_t fb_layernorm_bwd_mixed(fb_ctx* ctx, void* stream_, const void* x, int32_t x_bf16, const float* gamma, const float* beta,
                                      const float* mean, const float* rstd, const void* dy, int32_t dy_bf16, void* dx, float* dgamma,
                                      float* dbeta, int64_t d, int64_t n, int32_t act) {
  FB_CHECK_CTX(ctx);
  cudaStream_t stream = (cudaStream_t)stream_;
  FB_REQUIRE(d >= 1 && n >= 0, FB_ERR_SHAPE, "fb_layernorm_bwd_mixed: bad shape d=%lld n=%lld", (long long)d, (long long)n);
  FB_REQUIRE(fb_act_valid(act), FB_ERR_INVALID_ARG, "fb_layernorm_bwd_mixed: unknown activation %d", act);
  FB_REQUIRE((gamma == nullptr) == (beta == nullptr), FB_ERR_INVALID_ARG, "fb_layernorm_bwd_mixed: gamma and beta must both be given or both NULL");
  FB_REQUIRE((dgamma == nullptr) == (dbeta == nullptr), FB_ERR_INVALID_ARG, "fb_layernorm_bwd_mixed: dgamma and dbeta must both be given or both NULL");
  if (n == 0) {
    if (dgamma) {
      FB_CUDA(cudaMemsetAsync(dgamma, 0, d * sizeof(float), stream));
      FB_CUDA(cudaMemsetAsync(dbeta, 0, d * sizeof(float), stream));
    }
    return FB_OK;
  }
  FB_REQUIRE(x && mean && rstd && dy && (dx || dgamma), FB_ERR_INVALID_ARG, "fb_layernorm_bwd_mixed: NULL pointer");
  FB_REQUIRE(ln_low_ok(x, gamma, beta, dy, dx, d), FB_ERR_UNSUPPORTED, "fb_layernorm_bwd_mixed: needs 16-byte aligned arrays and a multiple of 8 up to 8192 features");
  const int64_t groups = fb_layernorm_bwd_groups(ctx->sm_count, d <= 1024 ? (n + 7) / 8 : n);
  float* part = nullptr;
  if (dgamma) {
    part = (float*)fb_scratch(ctx, stream, (size_t)(2 * groups * d) * sizeof(float));
    if (!part) return FB_ERR_ALLOC;
  }
  float *pg = part, *pb = part ? part + groups * d : nullptr;
  ln_low_dispatch(d, [&](auto V, auto T) {
    fb_act_kind(act, [&](auto k) {
      ln_flags(x_bf16 != 0, dy_bf16 != 0, [&](auto xb, auto db) {
        fb_launch(ln_bwd_low_kernel<V.value, T.value, k.value, xb.value, db.value>, (unsigned)groups, LN_THREADS, 0, stream, x, gamma, beta, mean, rstd, dy, dx, pg, pb, (int)d, n, act);
      });
    });
  });
  FB_LAUNCH_CHECK();
  if (dgamma) {
    fb_launch(fb_colreduce2_kernel, (unsigned)((d + 31) / 32), 256, 0, stream, pg, pb, dgamma, dbeta, groups, d);
    FB_LAUNCH_CHECK();
  }
  return FB_OK;
}

// ------------------------------------------------------------- LayerNorm backward without allocation ---
// Some callers of this library may not allocate device memory at all: a serving or training process whose whole
// memory budget was handed out at start-up, code running between the begin and end of a stream capture (where an
// allocation is an error), or a host runtime whose finaliser / callback threads must not trigger the implicit
// device synchronisation that cudaMalloc and cudaFree can cause.  For them the per-block dgamma / dbeta partials
// of the backward pass live in the fixed array below instead of the context arena.
//
// The array is part of the library image: every GPU that loads the library holds these 16 MiB until the process
// exits.  Its name is only a host-side handle; the device address is looked up once per device with
// cudaGetSymbolAddress while that device is current, and that pointer is what the kernels receive.
#include <mutex>

constexpr int64_t FB_LN_STATIC_FLOATS = int64_t(4) << 20;   // 4 Mi floats = 16 MiB
static __device__ __align__(256) float g_ln_static_scratch[FB_LN_STATIC_FLOATS];

namespace {
struct LnStaticDevice {
  float* scratch = nullptr;   // device address of g_ln_static_scratch on this device
  int sm_count = 0;
  bool ready = false;
};
constexpr int LN_STATIC_MAX_DEVICES = 64;
LnStaticDevice g_ln_static_dev[LN_STATIC_MAX_DEVICES];
std::mutex g_ln_static_mutex;
}  // namespace

FB_API int32_t fb_layernorm_bwd_noalloc(void* stream_, const float* x, const float* gamma, const float* beta,
                                        const float* mean, const float* rstd, const float* dy, float* dx,
                                        float* dgamma, float* dbeta, int64_t d, int64_t n, int32_t act) {
  cudaStream_t stream = (cudaStream_t)stream_;
  FB_REQUIRE(d >= 1 && n >= 0, FB_ERR_SHAPE, "fb_layernorm_bwd_noalloc: bad shape d=%lld n=%lld", (long long)d, (long long)n);
  FB_REQUIRE(fb_act_valid(act), FB_ERR_INVALID_ARG, "fb_layernorm_bwd_noalloc: unknown activation %d", act);
  FB_REQUIRE((gamma == nullptr) == (beta == nullptr), FB_ERR_INVALID_ARG, "fb_layernorm_bwd_noalloc: gamma and beta must both be given or both NULL");
  FB_REQUIRE((dgamma == nullptr) == (dbeta == nullptr), FB_ERR_INVALID_ARG, "fb_layernorm_bwd_noalloc: dgamma and dbeta must both be given or both NULL");
  // the partials need 2 * groups * d floats with at least one group
  FB_REQUIRE(dgamma == nullptr || 2 * d <= FB_LN_STATIC_FLOATS, FB_ERR_UNSUPPORTED,
             "fb_layernorm_bwd_noalloc: d = %lld exceeds the fixed scratch (at most %lld features when dgamma/dbeta are "
             "requested); use fb_layernorm_bwd",
             (long long)d, (long long)(FB_LN_STATIC_FLOATS / 2));
  int dev = -1;
  FB_CUDA(cudaGetDevice(&dev));
  FB_REQUIRE(dev >= 0 && dev < LN_STATIC_MAX_DEVICES, FB_ERR_UNSUPPORTED, "fb_layernorm_bwd_noalloc: device index %d not supported", dev);
  LnStaticDevice& sd = g_ln_static_dev[dev];
  {
    // first call on this device: resolve the device address of the array (the device is current here)
    std::lock_guard<std::mutex> lock(g_ln_static_mutex);
    if (!sd.ready) {
      float* p = nullptr;
      FB_CUDA(cudaGetSymbolAddress((void**)&p, g_ln_static_scratch));
      int sms = 0;
      FB_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
      sd.scratch = p;
      sd.sm_count = sms;
      sd.ready = true;
    }
  }
  if (n == 0) {
    if (dgamma) {
      FB_CUDA(cudaMemsetAsync(dgamma, 0, d * sizeof(float), stream));
      FB_CUDA(cudaMemsetAsync(dbeta, 0, d * sizeof(float), stream));
    }
    return FB_OK;
  }
  FB_REQUIRE(x && mean && rstd && dy && dx, FB_ERR_INVALID_ARG, "fb_layernorm_bwd_noalloc: NULL pointer");
  int64_t groups = fb_layernorm_bwd_groups(sd.sm_count, n);
  if (dgamma != nullptr) {
    const int64_t fit = FB_LN_STATIC_FLOATS / (2 * d);   // >= 1 by the check above
    if (groups > fit) groups = fit;
  }
  // Every block overwrites all d columns of its own partial rows before the reduction reads exactly
  // groups * d of them, so nothing left behind by an earlier call is ever read.
  // This entry point has no context and therefore no device error word to report a timed-out wait through, so it
  // keeps to the kernels that hold their rows in registers and wait on nothing (no shared-memory ring).
  return fb_layernorm_bwd_impl(stream, sd.sm_count, sd.scratch, groups, x, gamma, beta, mean, rstd, dy, dx, dgamma, dbeta,
                               d, n, act, nullptr, /*allow_ring=*/false);
}
