// Recurrence over LSTMCell / GRUCell: fused scan forward and BPTT backward.
//
// Layout: Julia x[in, T, B] is read as [B][T][in]; row (b, t) = b*T + t.  out[H, T, B] likewise.
// Forward:  (1) one GEMM over all T*B columns for the input projection Gx = x*Wi' + b,
//           (2) the time loop as one launch (rnn_seq.cuh).
// Backward: the reverse time loop as one launch (gate derivatives, dh_{t-1} = Wh' * dgates), then three GEMMs over all
//           T*B columns for dWi, dWh and dx.
// Where the hidden size does not fit the sequence kernels (beyond about 1180 units) a step is one launch forward and two
// backward, ordered by the stream.
#include <stdlib.h>

#include <type_traits>

#include <cuda_fp16.h>

#include "common.cuh"

namespace {

constexpr int RT = 256;      // threads per block
constexpr int BC = 64;       // batch columns per pass
constexpr int KC = 128;      // k values staged per pass
constexpr int HS = KC + 4;   // padded row stride of the staged h tile (float4-aligned, conflict-free)

// acc[r] += sum_k Ws[r][k] * v[b][k] for this thread's b and its quarter of every k-chunk.
//   Ws: shared [NR][kp] (kp = K rounded up to KC, zero padded); v: global rows of length K at stride ldv
//   (NULL = all zeros); vs: shared [BC][HS] staging tile.
template <int NR>
__device__ __forceinline__ void rows_times_vec(const float* __restrict__ Ws, int kp, const float* __restrict__ v,
                                               int64_t ldv, int K, int b0, int B, float* __restrict__ vs,
                                               float* acc) {
  const int b = threadIdx.x & (BC - 1), kq = threadIdx.x >> 6;
#pragma unroll
  for (int r = 0; r < NR; ++r) acc[r] = 0.0f;
  if (v == nullptr) return;
  for (int kc = 0; kc < kp; kc += KC) {
    __syncthreads();
    // stage v[b0 .. b0+BC)[kc .. kc+KC): 32 consecutive threads read 128 consecutive floats
    for (int e = threadIdx.x; e < BC * KC; e += RT) {
      const int bb = e / KC, kk = e % KC;
      const int gb = b0 + bb, gk = kc + kk;
      vs[bb * HS + kk] = (gb < B && gk < K) ? __ldg(v + (int64_t)gb * ldv + gk) : 0.0f;
    }
    __syncthreads();
    const float4* vrow = (const float4*)(vs + b * HS + kq * (KC / 4));
#pragma unroll 2
    for (int k4 = 0; k4 < KC / 16; ++k4) {
      const float4 hv = vrow[k4];
      const int kbase = kc + kq * (KC / 4) + k4 * 4;
#pragma unroll
      for (int r = 0; r < NR; ++r) {
        const float4 w = *(const float4*)(Ws + r * kp + kbase);
        acc[r] = fmaf(w.x, hv.x, acc[r]);
        acc[r] = fmaf(w.y, hv.y, acc[r]);
        acc[r] = fmaf(w.z, hv.z, acc[r]);
        acc[r] = fmaf(w.w, hv.w, acc[r]);
      }
    }
  }
}

// Sum the four k-quarter partials through shared memory: red[kq][b][r]; result for (b, r) in red[0][b][r].
template <int NR>
__device__ __forceinline__ void reduce_quarters(float* __restrict__ red, const float* acc) {
  const int b = threadIdx.x & (BC - 1), kq = threadIdx.x >> 6;
  __syncthreads();
#pragma unroll
  for (int r = 0; r < NR; ++r) red[(kq * BC + b) * (NR + 1) + r] = acc[r];
  __syncthreads();
  for (int e = threadIdx.x; e < BC * NR; e += RT) {
    const int bb = e / NR, r = e % NR;
    float s = 0.0f;
#pragma unroll
    for (int q = 0; q < 4; ++q) s += red[(q * BC + bb) * (NR + 1) + r];
    red[bb * (NR + 1) + r] = s;   // (0, bb, r) is only read by this thread in this pass
  }
  __syncthreads();
}

// Stage the NG*HU rows of Wh that belong to units [u0, u0+HU) into shared memory, zero padded to kp.
// Wh memory is [H (k)][NG*H (row)] (Julia Wh[NG*H, H]); row r = g*H + u.
template <int NG, int HU>
__device__ __forceinline__ void stage_w_rows(float* __restrict__ Ws, int kp, const float* __restrict__ Wh, int H, int u0) {
  for (int e = threadIdx.x; e < NG * HU * kp; e += RT) {
    const int k = e / (NG * HU), rr = e % (NG * HU);   // rr fastest: consecutive threads read neighbouring units
    const int g = rr / HU, u = rr % HU;
    float w = 0.0f;
    if (k < H && u0 + u < H) w = __ldg(Wh + (int64_t)k * (NG * H) + g * H + u0 + u);
    Ws[rr * kp + k] = w;
  }
}

// ------------------------------------------------------------------------------- LSTM forward step ---
template <int HU>
__global__ void __launch_bounds__(RT)
lstm_fwd_step_kernel(const float* __restrict__ Wh, const float* __restrict__ gx, const float* __restrict__ hprev,
                     int64_t ldh, const float* __restrict__ cprev, int64_t ldc, float* __restrict__ out_t,
                     int64_t ldo, float* __restrict__ gates_t, float* __restrict__ c_t, int64_t ldcache_g,
                     int64_t ldcache_c, float* __restrict__ hT, float* __restrict__ cT, int H, int B, int64_t ldgx) {
  extern __shared__ float sm[];
  const int kp = (H + KC - 1) / KC * KC;
  constexpr int NR = 4 * HU;
  float* Ws = sm;                         // [NR][kp]
  float* vs = Ws + NR * kp;               // [BC][HS]
  float* red = vs + BC * HS;              // [4][BC][NR+1]
  const int u0 = blockIdx.x * HU;
  stage_w_rows<4, HU>(Ws, kp, Wh, H, u0);
  for (int b0 = 0; b0 < B; b0 += BC) {
    float acc[NR];
    rows_times_vec<NR>(Ws, kp, hprev, ldh, H, b0, B, vs, acc);
    reduce_quarters<NR>(red, acc);
    for (int e = threadIdx.x; e < BC * HU; e += RT) {
      const int bb = e / HU, u = e % HU;
      const int gb = b0 + bb, gu = u0 + u;
      if (gb < B && gu < H) {
        const float* pre = red + bb * (NR + 1);
        const float* gxr = gx + (int64_t)gb * ldgx;
        const float zi = pre[0 * HU + u] + gxr[gu];
        const float zf = pre[1 * HU + u] + gxr[H + gu];
        const float zg = pre[2 * HU + u] + gxr[2 * H + gu];
        const float zo = pre[3 * HU + u] + gxr[3 * H + gu];
        const float ig = 1.0f / (1.0f + expf(-zi)), fg = 1.0f / (1.0f + expf(-zf));
        const float gg = tanhf(zg), og = 1.0f / (1.0f + expf(-zo));
        const float cp = cprev ? cprev[(int64_t)gb * ldc + gu] : 0.0f;
        const float cn = fg * cp + ig * gg;
        const float hn = og * tanhf(cn);
        out_t[(int64_t)gb * ldo + gu] = hn;
        if (gates_t) {
          float* gr = gates_t + (int64_t)gb * ldcache_g;
          gr[gu] = ig; gr[H + gu] = fg; gr[2 * H + gu] = gg; gr[3 * H + gu] = og;
        }
        c_t[(int64_t)gb * ldcache_c + gu] = cn;
        if (hT) { hT[(int64_t)gb * H + gu] = hn; cT[(int64_t)gb * H + gu] = cn; }
      }
    }
  }
}

// gate derivatives for step t, in place over the cached gates:
//   dh = dout_t + dh_rec; do = dh*tanh(c); dc += dh*o*(1-tanh(c)^2); di = dc*g; dg = dc*i; df = dc*c_prev
//   gates <- (di*i*(1-i), df*f*(1-f), dg*(1-g^2), do*o*(1-o)); dc_prev = dc*f
__global__ void __launch_bounds__(RT)
lstm_bwd_gates_kernel(float* __restrict__ gates_t, int64_t ldg, const float* __restrict__ c_t,
                      const float* __restrict__ c_prev, int64_t ldc, int64_t ldcp,
                      const float* __restrict__ dout_t, int64_t ldo, const float* __restrict__ dh_rec, int nparts,
                      float* __restrict__ dc, int H, int B) {
  const int64_t total = (int64_t)B * H;
  for (int64_t e = (int64_t)blockIdx.x * RT + threadIdx.x; e < total; e += (int64_t)gridDim.x * RT) {
    const int b = (int)(e / H), u = (int)(e % H);
    float* gr = gates_t + (int64_t)b * ldg;
    const float ig = gr[u], fg = gr[H + u], gg = gr[2 * H + u], og = gr[3 * H + u];
    const float tc = tanhf(c_t[(int64_t)b * ldc + u]);
    const float cp = c_prev ? c_prev[(int64_t)b * ldcp + u] : 0.0f;
    float dh = dout_t[(int64_t)b * ldo + u];
    if (dh_rec) for (int p = 0; p < nparts; ++p) dh += dh_rec[(int64_t)p * total + e];   // partials of Wh' * dgates
    const float d_o = dh * tc;
    const float dcc = dc[e] + dh * og * (1.0f - tc * tc);
    gr[u] = dcc * gg * ig * (1.0f - ig);
    gr[H + u] = dcc * cp * fg * (1.0f - fg);
    gr[2 * H + u] = dcc * ig * (1.0f - gg * gg);
    gr[3 * H + u] = d_o * og * (1.0f - og);
    dc[e] = dcc * fg;
  }
}

// -------------------------------------------------------------------------------- GRU forward step ---
// cache row layout per (b, t): [r (H)][z (H)][hc (H)][gh3 (H)]
template <int HU>
__global__ void __launch_bounds__(RT)
gru_fwd_step_kernel(const float* __restrict__ Wh, const float* __restrict__ gx, int64_t ldgx,
                    const float* __restrict__ hprev, int64_t ldh, float* __restrict__ out_t, int64_t ldo,
                    float* __restrict__ cache_t, int64_t ldcache, float* __restrict__ hT, int H, int B) {
  extern __shared__ float sm[];
  const int kp = (H + KC - 1) / KC * KC;
  constexpr int NR = 3 * HU;
  float* Ws = sm;
  float* vs = Ws + NR * kp;
  float* red = vs + BC * HS;
  const int u0 = blockIdx.x * HU;
  stage_w_rows<3, HU>(Ws, kp, Wh, H, u0);
  for (int b0 = 0; b0 < B; b0 += BC) {
    float acc[NR];
    rows_times_vec<NR>(Ws, kp, hprev, ldh, H, b0, B, vs, acc);
    reduce_quarters<NR>(red, acc);
    for (int e = threadIdx.x; e < BC * HU; e += RT) {
      const int bb = e / HU, u = e % HU;
      const int gb = b0 + bb, gu = u0 + u;
      if (gb < B && gu < H) {
        const float* pre = red + bb * (NR + 1);
        const float* gxr = gx + (int64_t)gb * ldgx;   // includes the bias
        const float gh3 = pre[2 * HU + u];
        const float r = 1.0f / (1.0f + expf(-(gxr[gu] + pre[u])));
        const float z = 1.0f / (1.0f + expf(-(gxr[H + gu] + pre[HU + u])));
        const float hc = tanhf(gxr[2 * H + gu] + r * gh3);
        const float hp = hprev ? hprev[(int64_t)gb * ldh + gu] : 0.0f;
        const float hn = (1.0f - z) * hc + z * hp;
        out_t[(int64_t)gb * ldo + gu] = hn;
        if (cache_t) {
          float* cr = cache_t + (int64_t)gb * ldcache;
          cr[gu] = r; cr[H + gu] = z; cr[2 * H + gu] = hc; cr[3 * H + gu] = gh3;
        }
        if (hT) hT[(int64_t)gb * H + gu] = hn;
      }
    }
  }
}

// GRU gate derivatives for step t.  Writes dgx_t = (da1, da2, da3) and dgh_t = (da1, da2, da3*r), and
// dh_direct = dh*z (the part of dh_{t-1} that does not go through Wh).
__global__ void __launch_bounds__(RT)
gru_bwd_gates_kernel(const float* __restrict__ cache_t, int64_t ldcache, const float* __restrict__ hprev, int64_t ldh,
                     const float* __restrict__ dout_t, int64_t ldo, const float* __restrict__ dh_rec, int nparts,
                     const float* __restrict__ dh_add, float* __restrict__ dgx_t, float* __restrict__ dgh_t, int64_t ldd,
                     float* __restrict__ dh_direct, int H, int B) {
  const int64_t total = (int64_t)B * H;
  for (int64_t e = (int64_t)blockIdx.x * RT + threadIdx.x; e < total; e += (int64_t)gridDim.x * RT) {
    const int b = (int)(e / H), u = (int)(e % H);
    const float* cr = cache_t + (int64_t)b * ldcache;
    const float r = cr[u], z = cr[H + u], hc = cr[2 * H + u], gh3 = cr[3 * H + u];
    const float hp = hprev ? hprev[(int64_t)b * ldh + u] : 0.0f;
    float dh = dout_t[(int64_t)b * ldo + u] + (dh_add ? dh_add[e] : 0.0f);
    if (dh_rec) for (int p = 0; p < nparts; ++p) dh += dh_rec[(int64_t)p * total + e];
    const float da3 = dh * (1.0f - z) * (1.0f - hc * hc);
    const float da2 = dh * (hp - hc) * z * (1.0f - z);
    const float da1 = da3 * gh3 * r * (1.0f - r);
    float* x_ = dgx_t + (int64_t)b * ldd;
    float* h_ = dgh_t + (int64_t)b * ldd;
    x_[u] = da1; x_[H + u] = da2; x_[2 * H + u] = da3;
    h_[u] = da1; h_[H + u] = da2; h_[2 * H + u] = da3 * r;
    dh_direct[e] = dh * z;
  }
}


// =============================================================================================
// Fast step kernels (H a multiple of 4 and small enough for shared memory): every global load of a step is a
// 128-bit load issued up front, so a step costs one memory round trip plus the FMA work.
// =============================================================================================

// pre[b][r] = sum_k W[r][k] * hprev[b][k] for the NG*4 gate rows of units [u0, u0+4) and a 64-wide batch chunk.
//   Ws: [NG*4][kp] (kp = H rounded up to 16), hs: [64][kp + 4], red: [4][64][NG*4 + 1].
//   On return red[b * (NR + 1) + r] holds the sums for this chunk.
template <int NG>
__device__ __forceinline__ void fast_gate_preacts(const float* __restrict__ Wh, const float* hprev, int64_t ldh,
                                                  int H, int B, int b0, int u0, int kp, float* __restrict__ Ws,
                                                  float* __restrict__ hs, float* __restrict__ red, bool load_w) {
  constexpr int NR = NG * 4;
  const int hs_ld = kp + 4;
  const int k4n = kp >> 2;
  if (load_w) {
    // W[k][g][u0 .. u0+3] is one 16-byte piece of the [H][NG*H] weight memory
    for (int e = threadIdx.x; e < kp * NG; e += RT) {
      const int k = e / NG, g = e % NG;
      float4 w = make_float4(0.f, 0.f, 0.f, 0.f);
      if (k < H) w = __ldg((const float4*)(Wh + (int64_t)k * (NG * H) + g * H + u0));
      Ws[(g * 4 + 0) * kp + k] = w.x;
      Ws[(g * 4 + 1) * kp + k] = w.y;
      Ws[(g * 4 + 2) * kp + k] = w.z;
      Ws[(g * 4 + 3) * kp + k] = w.w;
    }
  }
  if (hprev != nullptr) {
    for (int e = threadIdx.x; e < BC * k4n; e += RT) {
      const int bb = e / k4n, k4 = e % k4n;
      float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
      if (b0 + bb < B && 4 * k4 < H) v = __ldg((const float4*)(hprev + (int64_t)(b0 + bb) * ldh + 4 * k4));
      *(float4*)(hs + bb * hs_ld + 4 * k4) = v;
    }
  }
  __syncthreads();
  const int b = threadIdx.x & (BC - 1), kq = threadIdx.x >> 6;
  float acc[NR];
#pragma unroll
  for (int r = 0; r < NR; ++r) acc[r] = 0.0f;
  if (hprev != nullptr) {
    const int per = k4n >> 2;                       // float4 steps per quarter
    const float4* hrow = (const float4*)(hs + b * hs_ld) + kq * per;
    for (int i = 0; i < per; ++i) {
      const float4 hv = hrow[i];
      const int kbase = (kq * per + i) * 4;
#pragma unroll
      for (int r = 0; r < NR; ++r) {
        const float4 w = *(const float4*)(Ws + r * kp + kbase);
        acc[r] = fmaf(w.x, hv.x, acc[r]);
        acc[r] = fmaf(w.y, hv.y, acc[r]);
        acc[r] = fmaf(w.z, hv.z, acc[r]);
        acc[r] = fmaf(w.w, hv.w, acc[r]);
      }
    }
  }
#pragma unroll
  for (int r = 0; r < NR; ++r) red[(kq * BC + b) * (NR + 1) + r] = acc[r];
  __syncthreads();
  for (int e = threadIdx.x; e < BC * NR; e += RT) {
    const int bb = e / NR, r = e % NR;
    float sum = 0.0f;
#pragma unroll
    for (int q = 0; q < 4; ++q) sum += red[(q * BC + bb) * (NR + 1) + r];
    red[bb * (NR + 1) + r] = sum;
  }
  __syncthreads();
}

__global__ void __launch_bounds__(RT)
lstm_fwd_fast_kernel(const float* __restrict__ Wh, const float* __restrict__ gx, int64_t ldgx,
                     const float* __restrict__ hprev, int64_t ldh, const float* __restrict__ cprev, int64_t ldc,
                     float* __restrict__ out_t, int64_t ldo, float* __restrict__ gates_t, int64_t ldg,
                     float* __restrict__ c_t, int64_t ldct, float* __restrict__ hT, float* __restrict__ cT, int H, int B) {
  extern __shared__ __align__(16) float sm[];
  const int kp = (H + 15) & ~15;
  float* Ws = sm;
  float* hs = Ws + 16 * kp;
  float* red = hs + BC * (kp + 4);
  const int u0 = blockIdx.x * 4;
  for (int b0 = 0; b0 < B; b0 += BC) {
    if (b0 > 0) __syncthreads();
    fast_gate_preacts<4>(Wh, hprev, ldh, H, B, b0, u0, kp, Ws, hs, red, b0 == 0);
    const int bb = threadIdx.x >> 2, u = threadIdx.x & 3;     // 64 x 4 (batch, unit) pairs
    const int gb = b0 + bb, gu = u0 + u;
    if (gb < B && gu < H) {
      const float* pre = red + bb * 17;
      const float* gxr = gx + (int64_t)gb * ldgx;
      const float zi = pre[u] + gxr[gu], zf = pre[4 + u] + gxr[H + gu];
      const float zg = pre[8 + u] + gxr[2 * H + gu], zo = pre[12 + u] + gxr[3 * H + gu];
      const float ig = 1.0f / (1.0f + expf(-zi)), fg = 1.0f / (1.0f + expf(-zf));
      const float gg = tanhf(zg), og = 1.0f / (1.0f + expf(-zo));
      const float cp = cprev ? cprev[(int64_t)gb * ldc + gu] : 0.0f;
      const float cn = fg * cp + ig * gg;
      const float hn = og * tanhf(cn);
      out_t[(int64_t)gb * ldo + gu] = hn;
      if (gates_t) {
        float* gr = gates_t + (int64_t)gb * ldg;
        gr[gu] = ig; gr[H + gu] = fg; gr[2 * H + gu] = gg; gr[3 * H + gu] = og;
      }
      c_t[(int64_t)gb * ldct + gu] = cn;
      if (hT) { hT[(int64_t)gb * H + gu] = hn; cT[(int64_t)gb * H + gu] = cn; }
    }
  }
}

__global__ void __launch_bounds__(RT)
gru_fwd_fast_kernel(const float* __restrict__ Wh, const float* __restrict__ gx, int64_t ldgx,
                    const float* __restrict__ hprev, int64_t ldh, float* __restrict__ out_t, int64_t ldo,
                    float* __restrict__ cache_t, int64_t ldcache, float* __restrict__ hT, int H, int B) {
  extern __shared__ __align__(16) float sm[];
  const int kp = (H + 15) & ~15;
  float* Ws = sm;
  float* hs = Ws + 12 * kp;
  float* red = hs + BC * (kp + 4);
  const int u0 = blockIdx.x * 4;
  for (int b0 = 0; b0 < B; b0 += BC) {
    if (b0 > 0) __syncthreads();
    fast_gate_preacts<3>(Wh, hprev, ldh, H, B, b0, u0, kp, Ws, hs, red, b0 == 0);
    const int bb = threadIdx.x >> 2, u = threadIdx.x & 3;
    const int gb = b0 + bb, gu = u0 + u;
    if (gb < B && gu < H) {
      const float* pre = red + bb * 13;
      const float* gxr = gx + (int64_t)gb * ldgx;   // includes the bias
      const float gh3 = pre[8 + u];
      const float r = 1.0f / (1.0f + expf(-(gxr[gu] + pre[u])));
      const float z = 1.0f / (1.0f + expf(-(gxr[H + gu] + pre[4 + u])));
      const float hc = tanhf(gxr[2 * H + gu] + r * gh3);
      const float hp = hprev ? hprev[(int64_t)gb * ldh + gu] : 0.0f;
      const float hn = (1.0f - z) * hc + z * hp;
      out_t[(int64_t)gb * ldo + gu] = hn;
      if (cache_t) {
        float* cr = cache_t + (int64_t)gb * ldcache;
        cr[gu] = r; cr[H + gu] = z; cr[2 * H + gu] = hc; cr[3 * H + gu] = gh3;
      }
      if (hT) hT[(int64_t)gb * H + gu] = hn;
    }
  }
}

size_t fast_fwd_smem(int ng, int H) {
  const int kp = (H + 15) & ~15;
  return (size_t)(ng * 4 * kp + BC * (kp + 4) + 4 * BC * (ng * 4 + 1)) * sizeof(float);
}

// dh partials, 2-d decomposition: block (ub, rb, bz) computes, for units [64 ub, +64) and batch rows [64 bz, +64),
// the partial sum over gate rows r in [256 rb, +256):  part[rb][b][u] = sum_r dg[b][r] * Wm[u][r].
// Wm is the weight memory [H][R] (rows of R contiguous floats), so both operands stream as 128-bit loads.
constexpr int DH_U = 64, DH_R = 256, DH_LD = DH_R + 4;

__global__ void __launch_bounds__(RT)
rnn_bwd_dh2d_kernel(const float* __restrict__ Wh, const float* __restrict__ dg, int64_t ldg, float* __restrict__ part,
                    int H, int R, int B) {
  extern __shared__ __align__(16) float sm[];
  float* Ws = sm;                   // [64 u][DH_LD]
  float* Ds = Ws + DH_U * DH_LD;    // [64 b][DH_LD]
  const int u0 = blockIdx.x * DH_U, r0 = blockIdx.y * DH_R, b0 = blockIdx.z * BC;
  const bool vec = ((R & 3) == 0) && ((ldg & 3) == 0) && ((((uintptr_t)Wh | (uintptr_t)dg) & 15) == 0);
  for (int e = threadIdx.x; e < DH_U * (DH_R / 4); e += RT) {
    const int row = e / (DH_R / 4), c4 = e % (DH_R / 4);
    const int r = r0 + 4 * c4;
    float4 w = make_float4(0.f, 0.f, 0.f, 0.f), d = make_float4(0.f, 0.f, 0.f, 0.f);
    if (vec && r + 3 < R) {
      if (u0 + row < H) w = __ldg((const float4*)(Wh + (int64_t)(u0 + row) * R + r));
      if (b0 + row < B) d = __ldg((const float4*)(dg + (int64_t)(b0 + row) * ldg + r));
    } else {
      float wv[4] = {0.f, 0.f, 0.f, 0.f}, dv[4] = {0.f, 0.f, 0.f, 0.f};
      for (int i = 0; i < 4; ++i)
        if (r + i < R) {
          if (u0 + row < H) wv[i] = Wh[(int64_t)(u0 + row) * R + r + i];
          if (b0 + row < B) dv[i] = dg[(int64_t)(b0 + row) * ldg + r + i];
        }
      w = make_float4(wv[0], wv[1], wv[2], wv[3]);
      d = make_float4(dv[0], dv[1], dv[2], dv[3]);
    }
    *(float4*)(Ws + row * DH_LD + 4 * c4) = w;
    *(float4*)(Ds + row * DH_LD + 4 * c4) = d;
  }
  __syncthreads();
  // 16 x 16 threads, each a 4 x 4 tile: rows b = ty + 16 i, columns u = tx + 16 j
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  float acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0.0f;
  for (int c = 0; c < DH_R; c += 4) {
    float4 a[4], b[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) a[i] = *(const float4*)(Ds + (ty + 16 * i) * DH_LD + c);
#pragma unroll
    for (int j = 0; j < 4; ++j) b[j] = *(const float4*)(Ws + (tx + 16 * j) * DH_LD + c);
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        acc[i][j] = fmaf(a[i].x, b[j].x, acc[i][j]);
        acc[i][j] = fmaf(a[i].y, b[j].y, acc[i][j]);
        acc[i][j] = fmaf(a[i].z, b[j].z, acc[i][j]);
        acc[i][j] = fmaf(a[i].w, b[j].w, acc[i][j]);
      }
  }
  float* pp = part + (int64_t)blockIdx.y * B * H;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int gb = b0 + ty + 16 * i;
    if (gb >= B) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int gu = u0 + tx + 16 * j;
      if (gu < H) pp[(int64_t)gb * H + gu] = acc[i][j];
    }
  }
}

constexpr size_t DH2D_SMEM = (size_t)2 * DH_U * DH_LD * sizeof(float);

#include "rnn_seq.cuh"
#include "rnn_mma.cuh"

// hprev_all[(b, t)] = t == 0 ? h0[b] (or 0) : out[(b, t-1)]
__global__ void __launch_bounds__(RT)
shift_prev_kernel(const float* __restrict__ out, const float* __restrict__ h0, float* __restrict__ hprev_all, int H,
                  int64_t T, int64_t B) {
  fb_after_previous();
  const int64_t total = B * T * H;
  for (int64_t e = (int64_t)blockIdx.x * RT + threadIdx.x; e < total; e += (int64_t)gridDim.x * RT) {
    const int64_t row = e / H;
    const int u = (int)(e % H);
    const int64_t t = row % T, b = row / T;
    hprev_all[e] = t == 0 ? (h0 ? h0[b * H + u] : 0.0f) : out[e - H];
  }
}

// db[j] = sum over rows of dg[row][j]
int32_t colsum_rows(fb_ctx* ctx, cudaStream_t stream, const float* dg, float* db, int64_t rows, int64_t cols) {
  return fb_act_bwd_colsum(ctx, stream, FB_ACT_IDENTITY, dg, nullptr, nullptr, nullptr, db, rows, cols);
}

int pick_hu(int ng, int H, size_t smem_optin, size_t extra) {
  const int kp = (H + KC - 1) / KC * KC;
  const int cand[3] = {4, 2, 1};
  for (int i = 0; i < 3; ++i) {
    const size_t need = (size_t)(ng * cand[i]) * kp * 4 + extra + (size_t)4 * BC * (ng * cand[i] + 1) * 4;
    if (need <= smem_optin) return cand[i];
  }
  return 0;
}

size_t fwd_smem(int ng, int hu, int H) {
  const int kp = (H + KC - 1) / KC * KC;
  return (size_t)(ng * hu) * kp * 4 + (size_t)BC * HS * 4 + (size_t)4 * BC * (ng * hu + 1) * 4;
}

// FLUXB200_RNN_PERSIST = 0 keeps one launch per time step.
bool persistent_enabled() {
  static int on = -1;
  if (on < 0) {
    const char* e = getenv("FLUXB200_RNN_PERSIST");
    on = (e != nullptr && e[0] == '0') ? 0 : 1;
  }
  return on != 0;
}

// The blocks of the sequence kernels wait for one another's results (bounded), which needs every block resident at once.
// They are launched cooperatively, inside a stream capture too: the graph's kernel node keeps the attribute, so that two
// replays on two streams, or a replay beside other work, never hold half of the SMs each until the polls run out.

// Units and batch columns of a CTA of the sequence kernels, by the smallest modelled time of a step (us): the FMAs of the
// CTA's chunks at 60 % of the FMA rate (40 % for the narrow tiles), 0.8 per chunk (loads, reduction, gates), 1.3 for the
// exchange; backward the piece loads (60 B per cycle and SM) where they are longer than the FMAs.
struct SeqPlan {
  int ug, bg, nbg, grid;
  size_t smem;
};
bool plan_seq(const fb_ctx* ctx, int ng, int H, int64_t B, bool bwd, SeqPlan* best) {
  if (!persistent_enabled() || B > (1 << 20)) return false;
  double best_t = 1e30;
  for (int ug = 16; ug >= 8; ug /= 2)
    for (int bg = 16; bg >= 4; bg /= 2) {
      const int ugroups = (H + ug - 1) / ug;
      if (ugroups > ctx->sm_count) continue;
      const int64_t nch = (B + bg - 1) / bg;
      const int nbg = (int)(nch < ctx->sm_count / ugroups ? nch : ctx->sm_count / ugroups);
      const int64_t chunks = (nch + nbg - 1) / nbg;
      if (chunks > 64) continue;
      const size_t smem = bwd ? sq_bwd_smem(ng, ug, bg, H, (int)chunks) : sq_fwd_smem(ng, ug, bg, H, (int)chunks);
      if (smem > ctx->smem_optin) continue;
      const double fma = (double)ng * ug * bg * H / 128.0 / 1900.0 / (ug * bg >= 128 ? 0.6 : 0.4);
      const double load = bwd ? (double)ng * H * bg * 4.0 / 60.0 / 1900.0 : 0.0;
      const double t = chunks * ((fma > load ? fma : load) + 0.8) + 1.3;
      if (t < best_t) {
        best_t = t;
        best->ug = ug; best->bg = bg; best->nbg = nbg; best->grid = ugroups * nbg; best->smem = smem;
      }
    }
  return best_t < 1e30;
}

template <int NG, bool VEC>
const void* seq_fwd_kernel(int ug, int bg) {
  if (ug == 16) return bg == 16 ? (const void*)rnn_fwd_seq_kernel<NG, 16, 16, VEC> : bg == 8 ? (const void*)rnn_fwd_seq_kernel<NG, 16, 8, VEC> : (const void*)rnn_fwd_seq_kernel<NG, 16, 4, VEC>;
  return bg == 16 ? (const void*)rnn_fwd_seq_kernel<NG, 8, 16, VEC> : bg == 8 ? (const void*)rnn_fwd_seq_kernel<NG, 8, 8, VEC> : (const void*)rnn_fwd_seq_kernel<NG, 8, 4, VEC>;
}
template <int NG, bool VEC>
const void* seq_bwd_kernel(int ug, int bg) {
  if (ug == 16) return bg == 16 ? (const void*)rnn_bwd_seq_kernel<NG, 16, 16, VEC> : bg == 8 ? (const void*)rnn_bwd_seq_kernel<NG, 16, 8, VEC> : (const void*)rnn_bwd_seq_kernel<NG, 16, 4, VEC>;
  return bg == 16 ? (const void*)rnn_bwd_seq_kernel<NG, 8, 16, VEC> : bg == 8 ? (const void*)rnn_bwd_seq_kernel<NG, 8, 8, VEC> : (const void*)rnn_bwd_seq_kernel<NG, 8, 4, VEC>;
}

// The same for the tensor-core kernels (16 units x 8 or 16 columns a CTA).  Hidden sizes from 48 up to 512 (beyond, the fragments of the
// weights do not fit the registers), and sequences long enough to pay for the start (fragments, the buffer's fill).  The lines and the cost
// were drawn against the FMA kernels with an earlier backward kernel, which exchanged gate derivatives (us, forward and backward with bulk
// products): LSTM 512 x 64 columns, 256 steps 1650 + 2390 -> 890 + 1550; 4 steps 46 + 78 -> 39 + 75, 2 steps 35 + 67 -> 35 + 68, 1 step 25 +
// 48 -> 28 + 50; GRU 100 x 20, 3 steps 22 + 40 -> 27 + 43; LSTM 48 x 128, 50 steps 103 + 166 -> 97 + 148; 32 x 128, 20 steps 45 + 74 -> 48 + 76; 16
// x 1, 100 steps 143 + 167 -> 145 + 160.  The present backward kernel is no slower at any of 240 sizes tried above the lines (H 48 - 512, 1 - 512
// columns, 4 - 200 steps: by 1.0 at 48 to 1.46 at 400 units), also where its exchange of (H / 16)^2 blocks a step leaves L2: LSTM 512, 50 steps, 64, 130, 256 and 512
// columns 369, 885, 1260, 2489 -> 274, 651, 970, 2052; and where the buffer's fill is most of a short sequence: 130 columns, 4 steps 109 -> 81.
bool plan_mma(const fb_ctx* ctx, int ng, int H, int64_t B, int64_t T, bool bwd, SeqPlan* best) {
  if (!persistent_enabled() || B > (1 << 20) || H < 48 || H > 512 || T * H < 1536) return false;
  const int ugroups = (H + MQ_UG - 1) / MQ_UG;
  double best_t = 1e30;
  for (int bg = 16; bg >= 8; bg /= 2) {
    const int64_t nch = (B + bg - 1) / bg;
    const int nbg = (int)(nch < ctx->sm_count / ugroups ? nch : ctx->sm_count / ugroups);
    if (nbg < 1) continue;
    const int64_t chunks = (nch + nbg - 1) / nbg;
    if (chunks > MQ_CHUNKS) continue;
    const double t = chunks * (0.8 + 0.02 * bg) + 1.3;   // us of a step
    if (t < best_t) {
      best_t = t;
      best->ug = MQ_UG; best->bg = bg; best->nbg = nbg; best->grid = ugroups * nbg;
      best->smem = bwd ? mq_bwd_smem((int)chunks, bg) : mq_fwd_smem(ng, bg, H <= 128 ? 1 : H <= 256 ? 2 : 4, (int)chunks);
    }
  }
  return best_t < 1e30 && best->smem <= ctx->smem_optin;
}
template <int NG>
const void* mma_fwd_kernel(int bg, int H) {
  if (bg == 16) return H <= 128 ? (const void*)rnn_fwd_mma_kernel<NG, 16, 1> : H <= 256 ? (const void*)rnn_fwd_mma_kernel<NG, 16, 2> : (const void*)rnn_fwd_mma_kernel<NG, 16, 4>;
  return H <= 128 ? (const void*)rnn_fwd_mma_kernel<NG, 8, 1> : H <= 256 ? (const void*)rnn_fwd_mma_kernel<NG, 8, 2> : (const void*)rnn_fwd_mma_kernel<NG, 8, 4>;
}
template <int NG>
const void* mma_bwd_kernel(int bg, int H) {
  if (bg == 16) return H <= 128 ? (const void*)rnn_bwd_mma_kernel<NG, 16, 1> : H <= 256 ? (const void*)rnn_bwd_mma_kernel<NG, 16, 2> : (const void*)rnn_bwd_mma_kernel<NG, 16, 4>;
  return H <= 128 ? (const void*)rnn_bwd_mma_kernel<NG, 8, 1> : H <= 256 ? (const void*)rnn_bwd_mma_kernel<NG, 8, 2> : (const void*)rnn_bwd_mma_kernel<NG, 8, 4>;
}

// Launches the whole forward / backward time loop; FB_ERR_UNSUPPORTED (without a message) when the hidden size does not fit.
template <int NG>
int32_t launch_fwd_seq(fb_ctx* ctx, cudaStream_t stream, const float* Wh, const float* gx, const float* h0, const float* c0, float* out,
                       float* cache, float* cst, float* hT, float* cT, int H, int64_t B64, int64_t T64) {
  SeqPlan p;
  int B = (int)B64, T = (int)T64, cached = cache != nullptr ? 1 : 0;
  int32_t* dev_err = ctx->dev_error;
  if (plan_mma(ctx, NG, H, B64, T64, false, &p)) {
    const size_t bytes = (size_t)(T64 - 1) * mq_run(B64, p.bg, mq_pad(H)) * sizeof(float);
    const fb_temp mem(ctx, stream, bytes);
    if (bytes == 0 || mem.p != nullptr) {
      if (bytes != 0) FB_CUDA(cudaMemsetAsync(mem.p, 0xff, bytes, stream));
      const void* kern = mma_fwd_kernel<NG>(p.bg, H);
      float* ex = (float*)mem.p;
      void* args[] = {(void*)&Wh, (void*)&gx, (void*)&h0, (void*)&c0, (void*)&out, (void*)&cache, (void*)&cst, (void*)&cached, (void*)&hT,
                      (void*)&cT, (void*)&ex, (void*)&H, (void*)&B, (void*)&T, (void*)&p.nbg, (void*)&dev_err};
      FB_CUDA(fb_allow_smem(kern, ctx->smem_optin));
      FB_CUDA(cudaLaunchCooperativeKernel(kern, dim3((unsigned)p.grid), dim3(SQ_THREADS), args, p.smem, stream));
      FB_LAUNCH_CHECK();
      return FB_OK;
    }
  }
  if (!plan_seq(ctx, NG, H, B64, false, &p)) return FB_ERR_UNSUPPORTED;
  const bool vec = H % 4 == 0 && fb_aligned16(out) && fb_aligned16(h0);
  const void* kern = vec ? seq_fwd_kernel<NG, true>(p.ug, p.bg) : seq_fwd_kernel<NG, false>(p.ug, p.bg);
  if (T64 > 1) FB_CUDA(cudaMemsetAsync(out, 0xff, (size_t)(T64 * B64 * H) * sizeof(float), stream));
  int nbg = p.nbg;
  void* args[] = {(void*)&Wh, (void*)&gx, (void*)&h0, (void*)&c0, (void*)&out, (void*)&cache, (void*)&cst, (void*)&cached, (void*)&hT,
                  (void*)&cT, (void*)&H, (void*)&B, (void*)&T, (void*)&nbg, (void*)&dev_err};
  FB_CUDA(fb_allow_smem(kern, ctx->smem_optin));
  FB_CUDA(cudaLaunchCooperativeKernel(kern, dim3((unsigned)p.grid), dim3(SQ_THREADS), args, p.smem, stream));
  FB_LAUNCH_CHECK();
  return FB_OK;
}
template <int NG>
int32_t launch_bwd_seq(fb_ctx* ctx, cudaStream_t stream, const float* Wh, const float* keep, const float* cst, const float* s0,
                       const float* hout, const float* dout, const float* dhT, const float* dcT, float* dg, float* dgx, int H, int64_t B64,
                       int64_t T64) {
  SeqPlan p;
  int B = (int)B64, T = (int)T64;
  int32_t* dev_err = ctx->dev_error;
  if (plan_mma(ctx, NG, H, B64, T64, true, &p)) {
    const size_t slot = mq_part_run(B64, p.bg, H) * sizeof(float);
    int ring = T64 < MQ_RING || T64 * slot <= MQ_ALL_STEPS ? T : MQ_RING;
    const size_t bytes = T64 > 1 ? ring * slot : 0;
    const fb_temp mem(ctx, stream, bytes);
    if (bytes == 0 || mem.p != nullptr) {
      if (bytes != 0) FB_CUDA(cudaMemsetAsync(mem.p, 0xff, bytes, stream));
      const void* kern = mma_bwd_kernel<NG>(p.bg, H);
      float* ex = (float*)mem.p;
      void* args[] = {(void*)&Wh, (void*)&keep, (void*)&cst, (void*)&s0, (void*)&hout, (void*)&dout, (void*)&dhT, (void*)&dcT, (void*)&dg,
                      (void*)&dgx, (void*)&ex, (void*)&H, (void*)&B, (void*)&T, (void*)&p.nbg, (void*)&ring, (void*)&dev_err};
      FB_CUDA(fb_allow_smem(kern, mq_bwd_smem(MQ_CHUNKS, 16)));
      FB_CUDA(cudaLaunchCooperativeKernel(kern, dim3((unsigned)p.grid), dim3(SQ_THREADS), args, p.smem, stream));
      FB_LAUNCH_CHECK();
      return FB_OK;
    }
  }
  if (!plan_seq(ctx, NG, H, B64, true, &p)) return FB_ERR_UNSUPPORTED;
  const bool vec = NG * H % 4 == 0 && fb_aligned16(dg);
  const void* kern = vec ? seq_bwd_kernel<NG, true>(p.ug, p.bg) : seq_bwd_kernel<NG, false>(p.ug, p.bg);
  if (T64 > 1) FB_CUDA(cudaMemsetAsync(dg, 0xff, (size_t)(T64 * B64 * NG * H) * sizeof(float), stream));
  int nbg = p.nbg;
  void* args[] = {(void*)&Wh, (void*)&keep, (void*)&cst, (void*)&s0, (void*)&hout, (void*)&dout, (void*)&dhT, (void*)&dcT, (void*)&dg,
                  (void*)&dgx, (void*)&H, (void*)&B, (void*)&T, (void*)&nbg, (void*)&dev_err};
  FB_CUDA(fb_allow_smem(kern, ctx->smem_optin));
  FB_CUDA(cudaLaunchCooperativeKernel(kern, dim3((unsigned)p.grid), dim3(SQ_THREADS), args, p.smem, stream));
  FB_LAUNCH_CHECK();
  return FB_OK;
}

int32_t check_dims(const char* fn, int64_t in_dim, int64_t H, int64_t T, int64_t B) {
  FB_REQUIRE(in_dim >= 1 && H >= 1 && T >= 0 && B >= 0, FB_ERR_SHAPE, "%s: bad shape in=%lld H=%lld T=%lld B=%lld", fn,
             (long long)in_dim, (long long)H, (long long)T, (long long)B);
  FB_REQUIRE(H <= 16384 && B <= (1 << 24) && T <= (1 << 24), FB_ERR_SHAPE, "%s: dimension too large", fn);
  return FB_OK;
}

}  // namespace

FB_API int64_t fb_lstm_cache_bytes(int64_t in_dim, int64_t hidden, int64_t seq_len, int64_t batch) {
  (void)in_dim;
  // gates [B*T][4H] + cell states [B*T][H] + input projection [B*T][4H] (reused as scratch by the backward pass)
  return (int64_t)sizeof(float) * seq_len * batch * hidden * 9;
}

FB_API int64_t fb_gru_cache_bytes(int64_t in_dim, int64_t hidden, int64_t seq_len, int64_t batch) {
  (void)in_dim;
  // (r, z, hc, gh3) [B*T][4H] + input projection [B*T][3H] + recurrent-side gate derivatives [B*T][3H]
  // + shifted hidden states [B*T][H]
  return (int64_t)sizeof(float) * seq_len * batch * hidden * 11;
}

FB_API int32_t fb_lstm_fwd(fb_ctx* ctx, void* stream_, const float* Wi, const float* Wh, const float* b, const float* x,
                           const float* h0, const float* c0, float* out, float* hT, float* cT, void* cache,
                           int64_t in_dim, int64_t hidden, int64_t seq_len, int64_t batch) {
  FB_CHECK_CTX(ctx);
  cudaStream_t stream = (cudaStream_t)stream_;
  int32_t st = check_dims("fb_lstm_fwd", in_dim, hidden, seq_len, batch);
  if (st != FB_OK) return st;
  if (seq_len == 0 || batch == 0) return FB_OK;
  FB_REQUIRE(Wi && Wh && x && out, FB_ERR_INVALID_ARG, "fb_lstm_fwd: NULL pointer");
  FB_REQUIRE((hT == nullptr) == (cT == nullptr), FB_ERR_INVALID_ARG, "fb_lstm_fwd: hT and cT must both be given or both NULL");
  const int H = (int)hidden, B = (int)batch;
  const int64_t T = seq_len, rows = T * batch;
  float *gates, *cst, *gx;
  if (cache) {
    gates = (float*)cache;
    cst = gates + rows * 4 * H;
    gx = cst + rows * H;
  } else {
    float* ws = (float*)fb_scratch(ctx, stream, (size_t)(rows * 4 * H + 2 * (int64_t)B * H) * sizeof(float));
    if (!ws) return FB_ERR_ALLOC;
    gates = nullptr;
    gx = ws;
    cst = ws + rows * 4 * H;   // two [B][H] ping-pong cell buffers
  }
  // (1) input projection for every (b, t): gx[rows][4H] = x[rows][in] * Wi' + b
  fb_gemm_args a;
  a.A = x; a.lda = in_dim; a.a_mn_major = 0;
  a.B = Wi; a.ldb = 4 * hidden; a.b_mn_major = 1;
  a.C = gx; a.ldc = 4 * hidden; a.Z = nullptr; a.bias_n = b; a.bias_m = nullptr;
  a.M = rows; a.N = 4 * hidden; a.K = in_dim; a.act = FB_ACT_IDENTITY; a.accumulate = 0;
  st = fb_gemm_dispatch(ctx, stream, a, FB_PREC_DEFAULT);
  if (st != FB_OK) return st;
  // (2) time loop: one launch, or one per step where the hidden size does not fit
  st = launch_fwd_seq<4>(ctx, stream, Wh, gx, h0, c0, out, gates, cst, hT, cT, H, batch, T);
  if (st != FB_ERR_UNSUPPORTED) return st;
  const bool fast = (H % 4 == 0) && fb_aligned16(Wh) && fb_aligned16(out) && (!h0 || fb_aligned16(h0)) &&
                    fast_fwd_smem(4, H) <= ctx->smem_optin;
  const int hu = fast ? 4 : pick_hu(4, H, ctx->smem_optin, (size_t)BC * HS * 4);
  FB_REQUIRE(hu > 0, FB_ERR_UNSUPPORTED, "fb_lstm_fwd: hidden size %d does not fit the step kernel's shared memory", H);
  const size_t smem = fast ? fast_fwd_smem(4, H) : fwd_smem(4, hu, H);
  auto kern = hu == 4 ? lstm_fwd_step_kernel<4> : hu == 2 ? lstm_fwd_step_kernel<2> : lstm_fwd_step_kernel<1>;
  if (fast) FB_CUDA(fb_allow_smem(lstm_fwd_fast_kernel, ctx->smem_optin));
  else FB_CUDA(fb_allow_smem(kern, ctx->smem_optin));
  const unsigned grid = (unsigned)((H + hu - 1) / hu);
  const int64_t ldrow = T * H;       // stride between batch rows of out / cached c at a fixed t
  for (int64_t t = 0; t < T; ++t) {
    const float* hprev = t == 0 ? h0 : out + (t - 1) * H;
    const int64_t ldh = t == 0 ? H : ldrow;
    const float* cprev;
    int64_t ldcp;
    float* c_t;
    int64_t ldct;
    if (cache) {
      cprev = t == 0 ? c0 : cst + (t - 1) * H;
      ldcp = t == 0 ? H : ldrow;
      c_t = cst + t * H;
      ldct = ldrow;
    } else {
      cprev = t == 0 ? c0 : cst + ((t - 1) & 1) * (int64_t)B * H;
      ldcp = H;
      c_t = cst + (t & 1) * (int64_t)B * H;
      ldct = H;
    }
    float* g_t = gates ? gates + t * 4 * H : nullptr;
    float* hT_t = (t == T - 1) ? hT : nullptr;
    float* cT_t = (t == T - 1) ? cT : nullptr;
    if (fast)
      lstm_fwd_fast_kernel<<<grid, RT, smem, stream>>>(Wh, gx + t * 4 * H, T * 4 * H, hprev, ldh, cprev, ldcp, out + t * H, ldrow,
                                                       g_t, T * 4 * H, c_t, ldct, hT_t, cT_t, H, B);
    else
      kern<<<grid, RT, smem, stream>>>(Wh, gx + t * 4 * H, hprev, ldh, cprev, ldcp, out + t * H, ldrow, g_t, c_t, T * 4 * H, ldct,
                                       hT_t, cT_t, H, B, T * 4 * H);
    FB_LAUNCH_CHECK();
  }
  return FB_OK;
}

FB_API int32_t fb_lstm_bwd(fb_ctx* ctx, void* stream_, const float* Wi, const float* Wh, const float* x,
                           const float* h0, const float* c0, const float* out, const void* cache, const float* dout,
                           const float* dhT, const float* dcT,
                           float* dWi, float* dWh, float* db, float* dx, int64_t in_dim, int64_t hidden,
                           int64_t seq_len, int64_t batch) {
  FB_CHECK_CTX(ctx);
  cudaStream_t stream = (cudaStream_t)stream_;
  int32_t st = check_dims("fb_lstm_bwd", in_dim, hidden, seq_len, batch);
  if (st != FB_OK) return st;
  FB_REQUIRE(seq_len >= 1 && batch >= 1, FB_ERR_SHAPE, "fb_lstm_bwd: empty sequence or batch");
  FB_REQUIRE(Wi && Wh && x && out && cache && dout && dWi && dWh, FB_ERR_INVALID_ARG, "fb_lstm_bwd: NULL pointer");
  const int H = (int)hidden, B = (int)batch;
  const int64_t T = seq_len, rows = T * batch, ldrow = T * H;
  float* gates = (float*)cache;              // overwritten in place by the gate derivatives
  const float* cst = gates + rows * 4 * H;
  const int R = 4 * H;
  // the derivatives go over the input projection, which the backward pass does not need; the per-step kernels write them
  // over the gates
  float* dg = gates + rows * 5 * H;
  float* hprev_all = gates;
  st = launch_bwd_seq<4>(ctx, stream, Wh, gates, cst, c0, nullptr, dout, dhT, dcT, dg, nullptr, H, batch, T);
  if (st == FB_ERR_UNSUPPORTED) {
    dg = gates;
    hprev_all = gates + rows * 5 * H;
    const int nparts = (R + DH_R - 1) / DH_R;
    float* ws = (float*)fb_scratch(ctx, stream, (size_t)((1 + nparts) * (int64_t)B * H) * sizeof(float));
    if (!ws) return FB_ERR_ALLOC;
    float* dc = ws;                            // [B][H]
    float* parts = ws + (int64_t)B * H;        // [nparts][B][H] partial sums of Wh' * dgates
    if (dcT) FB_CUDA(cudaMemcpyAsync(dc, dcT, (size_t)B * H * sizeof(float), cudaMemcpyDeviceToDevice, stream));
    else FB_CUDA(cudaMemsetAsync(dc, 0, (size_t)B * H * sizeof(float), stream));
    FB_CUDA(cudaFuncSetAttribute(rnn_bwd_dh2d_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)DH2D_SMEM));
    const dim3 grid_dh((unsigned)((H + DH_U - 1) / DH_U), (unsigned)nparts, (unsigned)((B + BC - 1) / BC));
    int64_t eb = ((int64_t)B * H + RT - 1) / RT;
    if (eb > ctx->sm_count * 8) eb = ctx->sm_count * 8;
    for (int64_t t = T - 1; t >= 0; --t) {
      float* g_t = gates + t * 4 * H;
      const float* c_prev = t == 0 ? c0 : cst + (t - 1) * H;
      // recurrent dh entering step t: dhT at the last step, the partials of the step after it otherwise
      const float* dh_rec = (t == T - 1) ? dhT : parts;
      lstm_bwd_gates_kernel<<<(unsigned)eb, RT, 0, stream>>>(g_t, T * 4 * H, cst + t * H, c_prev, ldrow,
                                                             t == 0 ? (int64_t)H : ldrow, dout + t * H, ldrow, dh_rec,
                                                             (t == T - 1) ? 1 : nparts, dc, H, B);
      FB_LAUNCH_CHECK();
      if (t > 0) {
        rnn_bwd_dh2d_kernel<<<grid_dh, RT, DH2D_SMEM, stream>>>(Wh, g_t, T * 4 * H, parts, H, R, B);
        FB_LAUNCH_CHECK();
      }
    }
  } else if (st != FB_OK) {
    return st;
  }
  // bulk GEMMs over all T*B columns (dg is [rows][4H])
  fb_gemm_args a;
  a.Z = nullptr; a.bias_n = nullptr; a.bias_m = nullptr; a.act = FB_ACT_IDENTITY; a.accumulate = 0;
  // dWi memory [in][4H] = x^T dg
  a.A = x; a.lda = in_dim; a.a_mn_major = 1;
  a.B = dg; a.ldb = 4 * hidden; a.b_mn_major = 1;
  a.C = dWi; a.ldc = 4 * hidden; a.M = in_dim; a.N = 4 * hidden; a.K = rows;
  st = fb_gemm_dispatch(ctx, stream, a, FB_PREC_DEFAULT);
  if (st != FB_OK) return st;
  // dWh memory [H][4H] = hprev^T dg with hprev(b, t) = out(b, t-1) (h0 at t = 0); the shifted copy lives in
  // the region of the cache that the time loop has left.
  {
    int64_t sb = (rows * H + RT - 1) / RT;
    if (sb > (int64_t)ctx->sm_count * 16) sb = (int64_t)ctx->sm_count * 16;
    fb_launch(shift_prev_kernel, (unsigned)sb, RT, 0, stream, out, h0, hprev_all, H, T, batch);
    FB_LAUNCH_CHECK();
    a.A = hprev_all; a.lda = hidden; a.a_mn_major = 1;
    a.B = dg; a.ldb = 4 * hidden; a.b_mn_major = 1;
    a.C = dWh; a.ldc = 4 * hidden; a.M = hidden; a.N = 4 * hidden; a.K = rows;
    st = fb_gemm_dispatch(ctx, stream, a, FB_PREC_DEFAULT);
    if (st != FB_OK) return st;
  }
  a.accumulate = 0;
  if (db) {
    st = colsum_rows(ctx, stream, dg, db, rows, 4 * hidden);
    if (st != FB_OK) return st;
  }
  if (dx) {
    // dx[rows][in] = dg[rows][4H] * Wi (memory [in][4H]) ^T
    a.A = dg; a.lda = 4 * hidden; a.a_mn_major = 0;
    a.B = Wi; a.ldb = 4 * hidden; a.b_mn_major = 0;
    a.C = dx; a.ldc = in_dim; a.M = rows; a.N = in_dim; a.K = 4 * hidden;
    st = fb_gemm_dispatch(ctx, stream, a, FB_PREC_DEFAULT);
  }
  return st;
}

FB_API int32_t fb_gru_fwd(fb_ctx* ctx, void* stream_, const float* Wi, const float* Wh, const float* b, const float* x,
                          const float* h0, float* out, float* hT, void* cache, int64_t in_dim, int64_t hidden,
                          int64_t seq_len, int64_t batch) {
  FB_CHECK_CTX(ctx);
  cudaStream_t stream = (cudaStream_t)stream_;
  int32_t st = check_dims("fb_gru_fwd", in_dim, hidden, seq_len, batch);
  if (st != FB_OK) return st;
  if (seq_len == 0 || batch == 0) return FB_OK;
  FB_REQUIRE(Wi && Wh && x && out, FB_ERR_INVALID_ARG, "fb_gru_fwd: NULL pointer");
  const int H = (int)hidden, B = (int)batch;
  const int64_t T = seq_len, rows = T * batch, ldrow = T * H;
  float *cch = nullptr, *gx;
  if (cache) {
    cch = (float*)cache;
    gx = cch + rows * 4 * H;
  } else {
    gx = (float*)fb_scratch(ctx, stream, (size_t)(rows * 3 * H) * sizeof(float));
    if (!gx) return FB_ERR_ALLOC;
  }
  fb_gemm_args a;
  a.A = x; a.lda = in_dim; a.a_mn_major = 0;
  a.B = Wi; a.ldb = 3 * hidden; a.b_mn_major = 1;
  a.C = gx; a.ldc = 3 * hidden; a.Z = nullptr; a.bias_n = b; a.bias_m = nullptr;
  a.M = rows; a.N = 3 * hidden; a.K = in_dim; a.act = FB_ACT_IDENTITY; a.accumulate = 0;
  st = fb_gemm_dispatch(ctx, stream, a, FB_PREC_DEFAULT);
  if (st != FB_OK) return st;
  st = launch_fwd_seq<3>(ctx, stream, Wh, gx, h0, nullptr, out, cch, nullptr, hT, nullptr, H, batch, T);
  if (st != FB_ERR_UNSUPPORTED) return st;
  const bool fast = (H % 4 == 0) && fb_aligned16(Wh) && fb_aligned16(out) && (!h0 || fb_aligned16(h0)) &&
                    fast_fwd_smem(3, H) <= ctx->smem_optin;
  const int hu = fast ? 4 : pick_hu(3, H, ctx->smem_optin, (size_t)BC * HS * 4);
  FB_REQUIRE(hu > 0, FB_ERR_UNSUPPORTED, "fb_gru_fwd: hidden size %d does not fit the step kernel's shared memory", H);
  const size_t smem = fast ? fast_fwd_smem(3, H) : fwd_smem(3, hu, H);
  auto kern = hu == 4 ? gru_fwd_step_kernel<4> : hu == 2 ? gru_fwd_step_kernel<2> : gru_fwd_step_kernel<1>;
  if (fast) FB_CUDA(fb_allow_smem(gru_fwd_fast_kernel, ctx->smem_optin));
  else FB_CUDA(fb_allow_smem(kern, ctx->smem_optin));
  const unsigned grid = (unsigned)((H + hu - 1) / hu);
  for (int64_t t = 0; t < T; ++t) {
    const float* hprev = t == 0 ? h0 : out + (t - 1) * H;
    const int64_t ldh = t == 0 ? H : ldrow;
    float* c_t = cch ? cch + t * 4 * H : nullptr;
    float* hT_t = (t == T - 1) ? hT : nullptr;
    if (fast)
      gru_fwd_fast_kernel<<<grid, RT, smem, stream>>>(Wh, gx + t * 3 * H, T * 3 * H, hprev, ldh, out + t * H, ldrow, c_t, T * 4 * H,
                                                      hT_t, H, B);
    else
      kern<<<grid, RT, smem, stream>>>(Wh, gx + t * 3 * H, T * 3 * H, hprev, ldh, out + t * H, ldrow, c_t, T * 4 * H, hT_t, H, B);
    FB_LAUNCH_CHECK();
  }
  return FB_OK;
}

FB_API int32_t fb_gru_bwd(fb_ctx* ctx, void* stream_, const float* Wi, const float* Wh, const float* x,
                          const float* h0, const float* out, const void* cache, const float* dout, const float* dhT, float* dWi, float* dWh, float* db,
                          float* dx, int64_t in_dim, int64_t hidden, int64_t seq_len, int64_t batch) {
  FB_CHECK_CTX(ctx);
  cudaStream_t stream = (cudaStream_t)stream_;
  int32_t st = check_dims("fb_gru_bwd", in_dim, hidden, seq_len, batch);
  if (st != FB_OK) return st;
  FB_REQUIRE(seq_len >= 1 && batch >= 1, FB_ERR_SHAPE, "fb_gru_bwd: empty sequence or batch");
  FB_REQUIRE(Wi && Wh && x && out && cache && dout && dWi && dWh, FB_ERR_INVALID_ARG, "fb_gru_bwd: NULL pointer");
  const int H = (int)hidden, B = (int)batch;
  const int64_t T = seq_len, rows = T * batch, ldrow = T * H;
  const float* cch = (const float*)cache;          // [rows][4H]
  float* dgx = (float*)cache + rows * 4 * H;       // [rows][3H], over the input projection
  float* dgh = dgx + rows * 3 * H;                 // [rows][3H]
  const int R = 3 * H;
  st = launch_bwd_seq<3>(ctx, stream, Wh, cch, nullptr, h0, out, dout, dhT, nullptr, dgh, dgx, H, batch, T);
  if (st == FB_ERR_UNSUPPORTED) {
    const int nparts = (R + DH_R - 1) / DH_R;
    float* ws = (float*)fb_scratch(ctx, stream, (size_t)((1 + nparts) * (int64_t)B * H) * sizeof(float));
    if (!ws) return FB_ERR_ALLOC;
    float* dh_direct = ws;                     // dh * z, the part of dh_{t-1} that bypasses Wh
    float* parts = ws + (int64_t)B * H;        // [nparts][B][H] partial sums of Wh' * dgh
    FB_CUDA(cudaFuncSetAttribute(rnn_bwd_dh2d_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)DH2D_SMEM));
    const dim3 grid_dh((unsigned)((H + DH_U - 1) / DH_U), (unsigned)nparts, (unsigned)((B + BC - 1) / BC));
    int64_t eb = ((int64_t)B * H + RT - 1) / RT;
    if (eb > ctx->sm_count * 8) eb = ctx->sm_count * 8;
    for (int64_t t = T - 1; t >= 0; --t) {
      const float* hprev = t == 0 ? h0 : out + (t - 1) * H;
      const bool last = (t == T - 1);
      gru_bwd_gates_kernel<<<(unsigned)eb, RT, 0, stream>>>(cch + t * 4 * H, T * 4 * H, hprev, t == 0 ? (int64_t)H : ldrow,
                                                            dout + t * H, ldrow, last ? dhT : parts, last ? 1 : nparts,
                                                            last ? nullptr : dh_direct, dgx + t * 3 * H, dgh + t * 3 * H,
                                                            T * 3 * H, dh_direct, H, B);
      FB_LAUNCH_CHECK();
      if (t > 0) {
        rnn_bwd_dh2d_kernel<<<grid_dh, RT, DH2D_SMEM, stream>>>(Wh, dgh + t * 3 * H, T * 3 * H, parts, H, R, B);
        FB_LAUNCH_CHECK();
      }
    }
  } else if (st != FB_OK) {
    return st;
  }
  fb_gemm_args a;
  a.Z = nullptr; a.bias_n = nullptr; a.bias_m = nullptr; a.act = FB_ACT_IDENTITY; a.accumulate = 0;
  a.A = x; a.lda = in_dim; a.a_mn_major = 1;
  a.B = dgx; a.ldb = 3 * hidden; a.b_mn_major = 1;
  a.C = dWi; a.ldc = 3 * hidden; a.M = in_dim; a.N = 3 * hidden; a.K = rows;
  st = fb_gemm_dispatch(ctx, stream, a, FB_PREC_DEFAULT);
  if (st != FB_OK) return st;
  {
    float* hprev_all = dgh + rows * 3 * H;
    int64_t sb = (rows * H + RT - 1) / RT;
    if (sb > (int64_t)ctx->sm_count * 16) sb = (int64_t)ctx->sm_count * 16;
    fb_launch(shift_prev_kernel, (unsigned)sb, RT, 0, stream, out, h0, hprev_all, H, T, batch);
    FB_LAUNCH_CHECK();
    a.A = hprev_all; a.lda = hidden; a.a_mn_major = 1;
    a.B = dgh; a.ldb = 3 * hidden; a.b_mn_major = 1;
    a.C = dWh; a.ldc = 3 * hidden; a.M = hidden; a.N = 3 * hidden; a.K = rows;
    st = fb_gemm_dispatch(ctx, stream, a, FB_PREC_DEFAULT);
    if (st != FB_OK) return st;
  }
  a.accumulate = 0;
  if (db) {
    st = colsum_rows(ctx, stream, dgx, db, rows, 3 * hidden);
    if (st != FB_OK) return st;
  }
  if (dx) {
    a.A = dgx; a.lda = 3 * hidden; a.a_mn_major = 0;
    a.B = Wi; a.ldb = 3 * hidden; a.b_mn_major = 0;
    a.C = dx; a.ldc = in_dim; a.M = rows; a.N = in_dim; a.K = 3 * hidden;
    st = fb_gemm_dispatch(ctx, stream, a, FB_PREC_DEFAULT);
  }
  return st;
}
