// The time loop of an LSTM / GRU in one launch with the per-step products on the warp-level tensor cores (included by recurrent.cu
// behind rnn_seq.cuh, whose way of exchanging results it shares: words are polled in place until none is the empty pattern).
//
// CTA (unit group, batch group): 16 hidden units x BG = 8 or 16 columns.  Eight warps share k, and every warp keeps its
// part of the CTA's weight rows in registers for the whole launch, as mma.m16n8k16 fragments of two half-precision planes
// (W 2^s = hi + lo, 23 bits, with a power of two per row and 64 k-values).  Three products (lo hi, hi lo, hi hi) replace one Float32
// product; a warp's sum has at most 64 k-values (backward: sums of 64 are added up in Float32), then the warps' sums are added in Float32.
//
// Exchange.  A step's results go to a buffer of their own, as Float32 in the order of the fragments: [t][columns of a CTA][16 k-values]
// [8 columns][lane][4], so that a lane polls exactly the 16-byte pieces that it multiplies, a warp reads whole 512-byte runs
// and a CTA writes one: no shared memory and no barrier between the arrival of h and the product, and a warp waits for its own
// part only.  (The four k-values of a lane are neighbours; the order within a fragment is the same for both operands and does not
// matter to the sum.)  Read from `out`, whose rows lie T * H apart, the same pieces took 1.6 us of a step of 3.9 (L2: 8 rows of 64
// bytes a request, every row 512 KB from the next).  A column's scale is taken from the largest of the values that the warp
// multiplies, anew at every step and for every 64 of them: an element is held to 2^-23 of itself or 2^-39 of the largest of its 64.
// The initial state itself is multiplied in Float32.
//
// A warp that meets a weight or a value that is not finite, or an |h| of 16 or more (a GRU's initial state; |h| <= 1 otherwise), sums the
// products of that step in Float32 instead, from memory.
//
// What bounds it: T dependent steps (H 512, B 64: 5100 clocks): one store -> load flight through L2 (1200), the planes of h and 192 mma per
// SM partition at 8.7 clocks each (2250), the sum over the warps and the gates (1300).  FMA kernels 6.0 us a step, here 2.8.  Error against
// float64 is that of the FMA kernel.
#pragma once

constexpr int MQ_UG = 16, MQ_CHUNKS = 64;   // units of a CTA, its chunks of columns at most

__device__ __forceinline__ void mq_mma(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// two values -> their upper and lower halves
__device__ __forceinline__ void mq_split(float x, float y, uint32_t& hi, uint32_t& lo) {
  const __half2 h = __floats2half2_rn(x, y);
  const float2 f = __half22float2(h);
  const __half2 l = __floats2half2_rn(x - f.x, y - f.y);
  hi = *reinterpret_cast<const uint32_t*>(&h);
  lo = *reinterpret_cast<const uint32_t*>(&l);
}
// 2^s that puts a largest magnitude (its bits) into [2^14, 2^15), as s
__device__ __forceinline__ int mq_shift(uint32_t max_bits) {
  const int s = 141 - (int)(max_bits >> 23);
  return max_bits == 0 ? 0 : s > 126 ? 126 : s < -113 ? -113 : s;
}
__device__ __forceinline__ float mq_pow2(int s) { return __int_as_float((s + 127) << 23); }

// v * 2^e for |e| <= 252, in two factors
__device__ __forceinline__ float mq_unscale(float v, int e) {
  const int h = e >> 1;
  return v * mq_pow2(h) * mq_pow2(e - h);
}
__device__ __forceinline__ uint32_t mq_max4(uint32_t m, const uint4& x) {
  return max(m, max(max(x.x & 0x7fffffffu, x.y & 0x7fffffffu), max(x.z & 0x7fffffffu, x.w & 0x7fffffffu)));
}
// the largest magnitude (its bits) over the four lanes that share a row or column
__device__ __forceinline__ uint32_t mq_max_lanes(uint32_t m) {
  m = max(m, __shfl_xor_sync(0xffffffffu, m, 1));
  return max(m, __shfl_xor_sync(0xffffffffu, m, 2));
}
constexpr uint32_t MQ_INF = 0x7f800000u;
constexpr int MQ_MODERATE = 56;   // shifts whose powers of two can be multiplied with each other

// A fragments of KS k-steps: rows r and r + 8 of Ws, k-values k + 4 q .. of each step (k: the lane's first).  sh: the rows' shifts.
// Returns whether all of them are finite.
template <int KS>
__device__ __forceinline__ bool mq_load_a(const float* Ws, int ld, int r, int k, uint32_t (&hi)[KS][4], uint32_t (&lo)[KS][4], int (&sh)[2]) {
  uint32_t m[2] = {0u, 0u};
#pragma unroll
  for (int s = 0; s < KS; ++s)
#pragma unroll
    for (int i = 0; i < 2; ++i) m[i] = mq_max4(m[i], *(const uint4*)(Ws + (size_t)(r + 8 * i) * ld + k + 16 * s));
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    m[i] = mq_max_lanes(m[i]);
    sh[i] = mq_shift(m[i]);
  }
  const float s0 = mq_pow2(sh[0]), s8 = mq_pow2(sh[1]);
#pragma unroll
  for (int s = 0; s < KS; ++s) {
    const float4 x = *(const float4*)(Ws + (size_t)r * ld + k + 16 * s), y = *(const float4*)(Ws + (size_t)(r + 8) * ld + k + 16 * s);
    mq_split(x.x * s0, x.y * s0, hi[s][0], lo[s][0]);
    mq_split(y.x * s8, y.y * s8, hi[s][1], lo[s][1]);
    mq_split(x.z * s0, x.w * s0, hi[s][2], lo[s][2]);
    mq_split(y.z * s8, y.w * s8, hi[s][3], lo[s][3]);
  }
  return m[0] < MQ_INF && m[1] < MQ_INF;
}

// The pieces of one lane, k-steps ks .. ks + KS - 1 of a step's run (of `steps` of them), polled until all are there.  AGAIN asks only
// for those that were missing.
template <int NT, int KS>
struct MqPieces {
  uint4 v[NT][KS];
  static __device__ __forceinline__ bool empty(const uint4& x) {
    return (x.x == SQ_EMPTY) | (x.y == SQ_EMPTY) | (x.z == SQ_EMPTY) | (x.w == SQ_EMPTY);
  }
  template <bool AGAIN>
  __device__ __forceinline__ void load(const float* run, int ncols, int ks, int steps) {
    const int lane = threadIdx.x & 31;
    const float* p = run + (size_t)ks * (NT * 128) + 4 * lane;
#pragma unroll
    for (int s = 0; s < KS; ++s)
#pragma unroll
      for (int n = 0; n < NT; ++n) {
        if (AGAIN && !empty(v[n][s])) continue;
        uint4 x = make_uint4(0u, 0u, 0u, 0u);
        if (8 * n + (lane >> 2) < ncols && ks + s < steps) x = sq_peek4(p + (s * NT + n) * 128);
        v[n][s] = x;
      }
  }
  __device__ __forceinline__ bool complete() const {
    bool missing = false;
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
      for (int s = 0; s < KS; ++s) missing |= empty(v[n][s]);
    return !missing;
  }
  __device__ __forceinline__ bool wait(const float* run, int ncols, int ks, int steps, const int32_t* dev_err) {
    uint32_t spins = 0;
    while (!complete()) {
      if (++spins > SQ_POLL_LIMIT || ((spins & 255u) == 255u && *(const volatile int32_t*)dev_err != 0)) return false;
      load<true>(run, ncols, ks, steps);
    }
    return true;
  }
};
// words of a run: `batch` columns in whole groups of bg, k in whole k-steps
inline size_t mq_run(int64_t batch, int bg, int k) { return (size_t)((batch + bg - 1) / bg) * bg * k; }
inline int mq_pad(int n) { return (n + 15) / 16 * 16; }

// word (k-step ks, k-value gu of it, column gb) of a CTA's run
__device__ __forceinline__ void mq_publish(float* run, int bg, int ks, int gu, int gb, uint32_t w) {
  float* p = run + (size_t)ks * (bg * 16) + (gb >> 3) * 128 + (gb & 7) * 16 + gu;
  asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(w) : "memory");
}
__device__ __forceinline__ void mq_put4(float* p, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("st.relaxed.gpu.global.v4.u32 [%0], {%1, %2, %3, %4};" ::"l"(p), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}
// k-value k of column c of a run, as the exchange holds it
template <int NT>
__device__ __forceinline__ float mq_at(const float* run, int k, int c) {
  return __uint_as_float(sq_peek(run + (size_t)(k >> 4) * (NT * 128) + (c >> 3) * 128 + (c & 7) * 16 + (k & 15)));
}
__device__ __forceinline__ uint32_t mq_word(float v) {
  const uint32_t w = __float_as_uint(v);
  return w == SQ_EMPTY ? 0x7fffffffu : w;
}

inline size_t mq_fwd_smem(int ng, int bg, int ks, int chunks) {
  const size_t w = (size_t)ng * MQ_UG * (128 * ks + 4), red = (size_t)2 * 8 * bg * (MQ_UG + 1) * 4;
  return (w + red + (size_t)chunks * MQ_UG * bg) * 4;
}

// Arguments as for rnn_fwd_seq_kernel, and the exchange buffer (T - 1 runs); KS k-steps of 16 per warp: hidden sizes up to 128 KS.
template <int NG, int BG, int KS>
__global__ void __launch_bounds__(SQ_THREADS, 1)
rnn_fwd_mma_kernel(const float* __restrict__ Wh, const float* __restrict__ gx, const float* __restrict__ h0, const float* __restrict__ c0,
                   float* __restrict__ out, float* __restrict__ cache, float* __restrict__ cst, int cached, float* __restrict__ hT,
                   float* __restrict__ cT, float* ex, int H, int B, int T, int nbg, int32_t* dev_err) {
  constexpr int UG = MQ_UG, R = NG * UG, NT = BG / 8, LD = 128 * KS + 4, LU = UG + 1;
  extern __shared__ __align__(16) float sm[];
  float* Ws = sm;                            // [R][LD], until the initial state has been multiplied
  float4* red = (float4*)(Ws + R * LD);      // [2][8][BG][LU]: the gates of a unit and column side by side, in 16-byte accesses without conflicts
  float* cs = (float*)(red + 2 * 8 * BG * LU);   // [chunks][BG * UG]: LSTM c, GRU h
  const int ugroups = (H + UG - 1) / UG;
  const int u0 = ((int)blockIdx.x % ugroups) * UG, bgrp = (int)blockIdx.x / ugroups;
  const int nchunks = (B + BG - 1) / BG;
  const int64_t ldrow = (int64_t)T * H, ldgx = (int64_t)T * NG * H, ldc = (int64_t)T * 4 * H;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, q = lane & 3;
  const int gu = threadIdx.x % UG, gb = threadIdx.x / UG;   // gates: unit, column (threads below UG * BG)
  const int u = u0 + gu, ks0 = warp * KS, steps = (H + 15) / 16;
  const size_t run = (size_t)nchunks * BG * steps * 16;
  for (int e = threadIdx.x; e < R * 128 * KS; e += SQ_THREADS) {
    const int rr = e % R, k = e / R, g = rr / UG, uu = rr % UG;
    Ws[(size_t)rr * LD + k] = (k < H && u0 + uu < H) ? __ldg(Wh + (int64_t)k * (NG * H) + g * H + u0 + uu) : 0.0f;
  }
  for (int ch = bgrp, i = 0; ch < nchunks; ch += nbg, ++i) {
    const int b = ch * BG + gb;
    const float* s0 = NG == 4 ? c0 : h0;
    if (threadIdx.x < UG * BG) cs[i * UG * BG + threadIdx.x] = (s0 && b < B && u < H) ? s0[(int64_t)b * H + u] : 0.0f;
  }
  __syncthreads();
  uint32_t ahi[NG][KS][4], alo[NG][KS][4];
  int ash[NG][2];
  bool finite = true;
#pragma unroll
  for (int g = 0; g < NG; ++g) finite = mq_load_a<KS>(Ws, LD, g * UG + (lane >> 2), 16 * ks0 + 4 * q, ahi[g], alo[g], ash[g]) && finite;
  finite = __all_sync(0xffffffffu, finite);
  bool moderate = true;
#pragma unroll
  for (int g = 0; g < NG; ++g) moderate = moderate && abs(ash[g][0]) <= MQ_MODERATE && abs(ash[g][1]) <= MQ_MODERATE;
  int turn = 0;
  // The input projection of the next (step, chunk).  Asked for behind the poll: a poll that follows a load from DRAM returns no sooner
  // than that (LSTM 512, batch 64: the wait for h 2200 -> 1150 clocks).
  float gxn[NG];
  auto ahead = [&](int t, int ch) {
    const int b = ch * BG + gb;
    const bool there = threadIdx.x < UG * BG && b < B && u < H && t < T;
#pragma unroll
    for (int g = 0; g < NG; ++g) gxn[g] = there ? __ldg(gx + (int64_t)b * ldgx + (int64_t)t * NG * H + g * H + u) : 0.0f;
  };
  ahead(0, bgrp);
  for (int t = 0; t < T; ++t) {
    for (int ch = bgrp, ci = 0; ch < nchunks; ch += nbg, ++ci, turn ^= 1) {
      const int b0 = ch * BG, nb = B - b0 < BG ? B - b0 : BG;
      const int b = b0 + gb;
      const bool mine = threadIdx.x < UG * BG && gb < nb && u < H;
      float gxv[NG];
#pragma unroll
      for (int g = 0; g < NG; ++g) gxv[g] = gxn[g];
      float pre[NG];
#pragma unroll
      for (int g = 0; g < NG; ++g) pre[g] = 0.0f;
      if (t > 0) {
        const float* src = ex + (size_t)(t - 1) * run + (size_t)ch * (BG * 16) * steps;
        MqPieces<NT, KS> pc;
        pc.template load<false>(src, nb, ks0, steps);
        const bool ok = pc.wait(src, nb, ks0, steps, dev_err);
        ahead(ch + nbg < nchunks ? t : t + 1, ch + nbg < nchunks ? ch + nbg : bgrp);
        float acc[NG][NT][4];
#pragma unroll
        for (int g = 0; g < NG; ++g)
#pragma unroll
          for (int n = 0; n < NT; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[g][n][e] = 0.0f;
        int hsh[NT];
        bool small = finite;
#pragma unroll
        for (int n = 0; n < NT; ++n) {
          uint32_t m = 0u;
#pragma unroll
          for (int s = 0; s < KS; ++s) m = mq_max4(m, pc.v[n][s]);
          m = mq_max_lanes(m);
          hsh[n] = mq_shift(m);
          small = small && m < 0x41800000u;   // 16
        }
        float4* rw = red + (turn * 8 + warp) * BG * LU + (lane >> 2);
        auto put = [&](int n, int e) {   // column 8 n + 2 q + (e & 1), unit (lane >> 2) + 8 (e >> 1)
          rw[(8 * n + 2 * q + (e & 1)) * LU + 8 * (e >> 1)] = make_float4(acc[0][n][e], acc[1][n][e], acc[2][n][e], NG == 4 ? acc[NG - 1][n][e] : 0.0f);
        };
        if (__all_sync(0xffffffffu, small || !ok)) {
          // The cross terms of all k-steps first: an add into the accumulator truncates, so the fewer behind the large terms the
          // better.  Product by product over all accumulators, so that an mma does not follow the one that it adds to.
          uint32_t hi[KS][NT][2];
#pragma unroll
          for (int s = 0; s < KS; ++s) {
            uint32_t lo[NT][2];
#pragma unroll
            for (int n = 0; n < NT; ++n) {
              const uint4 x = pc.v[n][s];
              const float sc = mq_pow2(hsh[n]);
              mq_split(__uint_as_float(x.x) * sc, __uint_as_float(x.y) * sc, hi[s][n][0], lo[n][0]);
              mq_split(__uint_as_float(x.z) * sc, __uint_as_float(x.w) * sc, hi[s][n][1], lo[n][1]);
            }
#pragma unroll
            for (int n = 0; n < NT; ++n)
#pragma unroll
              for (int g = 0; g < NG; ++g) mq_mma(acc[g][n], alo[g][s], hi[s][n][0], hi[s][n][1]);
#pragma unroll
            for (int n = 0; n < NT; ++n)
#pragma unroll
              for (int g = 0; g < NG; ++g) mq_mma(acc[g][n], ahi[g][s], lo[n][0], lo[n][1]);
          }
#pragma unroll
          for (int s = 0; s < KS; ++s)
#pragma unroll
            for (int n = 0; n < NT; ++n)
#pragma unroll
              for (int g = 0; g < NG; ++g) mq_mma(acc[g][n], ahi[g][s], hi[s][n][0], hi[s][n][1]);
          // columns 2 q and 2 q + 1 were scaled by the lanes that hold them
#pragma unroll
          for (int n = 0; n < NT; ++n) {
            const int c0 = __shfl_sync(0xffffffffu, hsh[n], 8 * q), c1 = __shfl_sync(0xffffffffu, hsh[n], 8 * q + 4);
            if (moderate && (c0 <= MQ_MODERATE) & (c1 <= MQ_MODERATE)) {   // (c >= 10, as |h| < 16) factors that no product of them leaves the range with
              const float f0 = mq_pow2(-c0), f1 = mq_pow2(-c1);
#pragma unroll
              for (int e = 0; e < 4; ++e) {
#pragma unroll
                for (int g = 0; g < NG; ++g) acc[g][n][e] *= mq_pow2(-ash[g][e >> 1]) * ((e & 1) ? f1 : f0);
                put(n, e);
              }
            } else {
#pragma unroll
              for (int e = 0; e < 4; ++e) {
#pragma unroll
                for (int g = 0; g < NG; ++g) acc[g][n][e] = mq_unscale(acc[g][n][e], -(ash[g][e >> 1] + ((e & 1) ? c1 : c0)));
                put(n, e);
              }
            }
          }
        } else {
          for (int k = 16 * ks0; k < 16 * (ks0 + KS) && k < H; ++k)
#pragma unroll
            for (int n = 0; n < NT; ++n)
#pragma unroll
              for (int e = 0; e < 4; ++e) {
                const int c = 8 * n + 2 * q + (e & 1), uu = (lane >> 2) + 8 * (e >> 1);
                const float h = c < nb ? mq_at<NT>(src, k, c) : 0.0f;
#pragma unroll
                for (int g = 0; g < NG; ++g)
                  if (u0 + uu < H) acc[g][n][e] = fmaf(__ldg(Wh + (int64_t)k * (NG * H) + g * H + u0 + uu), h, acc[g][n][e]);
              }
#pragma unroll
          for (int n = 0; n < NT; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) put(n, e);
        }
        // One barrier a step: sums of the step after next come behind the next one's, where this step's have been read.
        if (!__syncthreads_and(ok ? 1 : 0)) {
          if (threadIdx.x == 0) atomicCAS(dev_err, 0, 3002);
          return;
        }
        if (mine) {
#pragma unroll
          for (int w = 0; w < 8; ++w) {
            const float4 s = red[((turn * 8 + w) * BG + gb) * LU + gu];
            pre[0] += s.x;
            pre[1] += s.y;
            pre[2] += s.z;
            if (NG == 4) pre[NG - 1] += s.w;
          }
        }
      } else {
        ahead(ch + nbg < nchunks ? t : t + 1, ch + nbg < nchunks ? ch + nbg : bgrp);
        if (h0 != nullptr && mine) {
#pragma unroll 4
          for (int k = 0; k < H; ++k) {
            const float h = __ldg(h0 + (int64_t)b * H + k);
#pragma unroll
            for (int g = 0; g < NG; ++g) pre[g] = fmaf(Ws[(g * UG + gu) * LD + k], h, pre[g]);
          }
        }
      }
      if (mine) {
        float hn, cn = 0.0f;
        float4 keep;
        float* c = cs + ci * UG * BG + threadIdx.x;
        if (NG == 4) {
          const float zi = pre[0] + gxv[0], zf = pre[1] + gxv[1], zg = pre[2] + gxv[2], zo = pre[NG - 1] + gxv[NG - 1];
          const float ig = 1.0f / (1.0f + expf(-zi)), fg = 1.0f / (1.0f + expf(-zf));
          const float gg = tanhf(zg), og = 1.0f / (1.0f + expf(-zo));
          cn = fg * *c + ig * gg;
          *c = cn;
          hn = og * tanhf(cn);
          keep = make_float4(ig, fg, gg, og);
        } else {
          const float gh3 = pre[2];
          const float r = 1.0f / (1.0f + expf(-(gxv[0] + pre[0])));
          const float z = 1.0f / (1.0f + expf(-(gxv[1] + pre[1])));
          const float hc = tanhf(gxv[2] + r * gh3);
          hn = (1.0f - z) * hc + z * *c;
          *c = hn;
          keep = make_float4(r, z, hc, gh3);
        }
        if (t + 1 < T) mq_publish(ex + (size_t)t * run + (size_t)ch * (BG * 16) * steps, BG, u0 / 16, gu, gb, mq_word(hn));
        out[(int64_t)t * H + (int64_t)b * ldrow + u] = hn;
        if (cache) {
          float* gr = cache + (int64_t)t * 4 * H + (int64_t)b * ldc;
          gr[u] = keep.x; gr[H + u] = keep.y; gr[2 * H + u] = keep.z; gr[3 * H + u] = keep.w;
        }
        if (NG == 4 && cached) cst[(int64_t)t * H + (int64_t)b * ldrow + u] = cn;
        if (t == T - 1 && hT) {
          hT[(int64_t)b * H + u] = hn;
          if (NG == 4) cT[(int64_t)b * H + u] = cn;
        }
      } else if (t + 1 < T && threadIdx.x < UG * BG && gb < nb) {
        mq_publish(ex + (size_t)t * run + (size_t)ch * (BG * 16) * steps, BG, u0 / 16, gu, gb, 0u);   // (units that do not exist)
      }
    }
  }
}

// Backward.  The same CTAs; a CTA turns dh_t of its units into its own gate derivatives dg_t (NG * 16 rows x BG columns, one k-step per
// gate) and multiplies them at once with its rows of Wh', for ALL units: a warp owns the 16-unit groups warp, warp + 8, ... and keeps
// their fragments in registers.  What travels is the product: each group's CTA gets one partial sum per producer, polled in place
// and added up in the producers' order.  (With dg itself exchanged a CTA read 4 H words per column and step, 128 KB at H 512, and cut
// all of them into planes.)  H 512, B 64, T 256: 4.8 -> 3.35 us a step; what bounds it: 192 mma per SM partition (0.9 us), the sums'
// way through L2 (32 KB out, in and reset per CTA: 1.3 us), gates and planes (0.5 us).
//
// Exchange: [slot][chunk][consumer group][producer group][BG / 8][lane][4], a lane's accumulators as it holds them.  Up to MQ_ALL_STEPS
// bytes every step has a slot of its own.  Beyond, MQ_RING slots take the steps in turn, so that they stay in L2: a consumer puts the
// empty pattern back over what it has read, and the slot is written again MQ_RING steps later.  That the pattern is there by then: every
// thread fences in every MQ_FENCE-th step (steps count down), behind the barrier that follows the resets and ahead of the one before
// the CTA sends.  A reset of step s lies before its CTA's fence of a step f, s >= f > s - MQ_FENCE, and so before what that CTA sends in f;
// who has received that fences in step f - MQ_FENCE, before it writes to the same slot in step s + 1 - MQ_RING.
// (Rings of 4, 8 and 16: 885, 847, 868 us at B 64; 1746, 1677, 1637 at B 128.  Resets behind the products or by bulk copies delay what is
// sent: 910 - 1040 us.)
constexpr int MQ_FENCE = 6, MQ_RING = 2 * MQ_FENCE;
constexpr size_t MQ_ALL_STEPS = (size_t)32 << 20;   // bytes up to which every step gets a slot of its own, and nothing is reset
constexpr int MQ_BAD = 1000;   // in the place of a column's shift: a value of it is not finite

inline size_t mq_part_run(int64_t batch, int bg, int H) {
  const size_t groups = (size_t)(H + MQ_UG - 1) / MQ_UG;
  return (size_t)((batch + bg - 1) / bg) * groups * groups * (MQ_UG * bg);
}
inline size_t mq_bwd_smem(int chunks, int bg) { return (size_t)chunks * MQ_UG * bg * sizeof(float); }   // beside the kernel's own

template <int NG, int BG, int MT>
__global__ void __launch_bounds__(SQ_THREADS, 1)
rnn_bwd_mma_kernel(const float* __restrict__ Wh, const float* __restrict__ keep, const float* __restrict__ cst,
                   const float* __restrict__ s0, const float* __restrict__ hout, const float* __restrict__ dout,
                   const float* __restrict__ dhT, const float* __restrict__ dcT, float* __restrict__ dg, float* __restrict__ dgx,
                   float* ex, int H, int B, int T, int nbg, int ring, int32_t* dev_err) {
  constexpr int UG = MQ_UG, NT = BG / 8, BLOCK = UG * BG;
  constexpr int PIECES = 32 * NT, GRP = SQ_THREADS / PIECES, PER = 8 * MT / GRP;   // GRP sets of threads share the producers
  constexpr int LS = 20;                          // words of the sums per 16: the gates' threads read them without bank conflicts
  __shared__ __align__(16) float sums[GRP][NT][8 * LS];
  __shared__ __align__(16) uint4 frag[NG][NT][32];   // {hi, hi, lo, lo} of a lane's four k-values
  __shared__ float dval[BG][NG * UG];             // the values themselves
  __shared__ int csh[BG];                         // the columns' shifts
  extern __shared__ float carry[];                // [chunks][UG * BG]: LSTM dc, GRU dh * z
  const int K = NG * H;
  const int ugroups = (H + UG - 1) / UG;
  const int ug = (int)blockIdx.x % ugroups, bgrp = (int)blockIdx.x / ugroups, u0 = ug * UG;
  const int nchunks = (B + BG - 1) / BG;
  const int64_t ldd = (int64_t)T * K;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, q = lane & 3;
  const int gu = threadIdx.x % UG, gb = threadIdx.x / UG;
  const int u = u0 + gu;
  const bool gates = threadIdx.x < BLOCK;
  const size_t run = (size_t)nchunks * ugroups * ugroups * BLOCK;
  for (int ch = bgrp, i = 0; ch < nchunks; ch += nbg, ++i) {
    const int b = ch * BG + gb;
    if (gates) carry[i * BLOCK + threadIdx.x] = (NG == 4 && dcT && b < B && u < H) ? dcT[(int64_t)b * H + u] : 0.0f;
  }
  // fragments of Wh': rows (lane >> 2) and 8 more of each group, this CTA's NG * 16 k-values
  uint32_t ahi[MT][NG][4], alo[MT][NG][4];
  int ash[MT][2];
  bool finite = true, moderate = true;
#pragma unroll
  for (int m = 0; m < MT; ++m) {
    float v[2][NG][4];
    uint32_t mx[2] = {0u, 0u};
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int row = (warp + 8 * m) * UG + (lane >> 2) + 8 * i;
#pragma unroll
      for (int g = 0; g < NG; ++g)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          v[i][g][e] = (row < H && u0 + 4 * q + e < H) ? __ldg(Wh + (int64_t)row * K + g * H + u0 + 4 * q + e) : 0.0f;
          mx[i] = max(mx[i], __float_as_uint(v[i][g][e]) & 0x7fffffffu);
        }
      mx[i] = mq_max_lanes(mx[i]);
      ash[m][i] = mq_shift(mx[i]);
      moderate = moderate && abs(ash[m][i]) <= MQ_MODERATE;
      const float sc = mq_pow2(ash[m][i]);
#pragma unroll
      for (int g = 0; g < NG; ++g) {
        mq_split(v[i][g][0] * sc, v[i][g][1] * sc, ahi[m][g][i], alo[m][g][i]);
        mq_split(v[i][g][2] * sc, v[i][g][3] * sc, ahi[m][g][2 + i], alo[m][g][2 + i]);
      }
    }
    finite = finite && mx[0] < MQ_INF && mx[1] < MQ_INF;
  }
  __syncthreads();
  // What a step reads of its own units, asked for a step ahead and behind the poll (as in the forward kernel).  No branch around the loads:
  // where paths meet, the compiler waits for what is on its way.
  float nk[4], nct = 0.0f, nsp = 0.0f, ndh = 0.0f;
  auto ahead = [&](int t, int ch) {
    const int b = ch * BG + gb;
    const bool there = gates && b < B && u < H && t >= 0;
    const int64_t row = there ? (int64_t)b * T + t : 0;
    const float *kr = keep + row * 4 * H + u, *prev = NG == 4 ? cst : hout;   // c_{t-1} or h_{t-1}
#pragma unroll
    for (int i = 0; i < 4; ++i) nk[i] = there ? __ldg(kr + i * H) : 0.0f;
    if (NG == 4) nct = there ? __ldg(cst + row * H + u) : 0.0f;
    nsp = there && t > 0 ? __ldg(prev + (row - 1) * H + u) : 0.0f;
    ndh = there ? __ldg(dout + row * H + u) : 0.0f;
  };
  ahead(T - 1, bgrp);
  const int grp = threadIdx.x / PIECES, piece = threadIdx.x % PIECES;
  for (int t = T - 1; t >= 0; --t) {
    for (int ch = bgrp, ci = 0; ch < nchunks; ch += nbg, ++ci) {
      const int b0 = ch * BG, nb = B - b0 < BG ? B - b0 : BG;
      const int b = b0 + gb;
      const bool mine = gates && gb < nb && u < H;
      const float k0 = nk[0], k1 = nk[1], k2 = nk[2], k3 = nk[3], ct = nct;
      float sp = nsp, dh = ndh;
      if (t == 0 && s0 && mine) sp = __ldg(s0 + (int64_t)b * H + u);
      if (t == T - 1 && dhT && mine) dh += __ldg(dhT + (int64_t)b * H + u);
      if (t < T - 1) {
        float* src = ex + (size_t)((t + 1) % ring) * run + ((size_t)ch * ugroups + ug) * ugroups * BLOCK + 4 * piece;
        uint4 v[PER];
        bool missing = false;
#pragma unroll
        for (int i = 0; i < PER; ++i) {
          const int p = grp + GRP * i;
          v[i] = p < ugroups ? sq_peek4(src + (size_t)p * BLOCK) : make_uint4(0u, 0u, 0u, 0u);
        }
#pragma unroll
        for (int i = 0; i < PER; ++i) missing |= MqPieces<1, 1>::empty(v[i]);
        bool ok = true;
        uint32_t spins = 0;
        while (missing) {
          if (++spins > SQ_POLL_LIMIT || ((spins & 255u) == 255u && *(const volatile int32_t*)dev_err != 0)) {
            ok = false;
            break;
          }
          missing = false;
#pragma unroll
          for (int i = 0; i < PER; ++i)
            if (MqPieces<1, 1>::empty(v[i])) v[i] = sq_peek4(src + (size_t)(grp + GRP * i) * BLOCK);
#pragma unroll
          for (int i = 0; i < PER; ++i) missing |= MqPieces<1, 1>::empty(v[i]);
        }
        float4 s = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
        for (int i = 0; i < PER; ++i) {
          s.x += __uint_as_float(v[i].x);
          s.y += __uint_as_float(v[i].y);
          s.z += __uint_as_float(v[i].z);
          s.w += __uint_as_float(v[i].w);
          if (ring < T && grp + GRP * i < ugroups) mq_put4(src + (size_t)(grp + GRP * i) * BLOCK, SQ_EMPTY, SQ_EMPTY, SQ_EMPTY, SQ_EMPTY);
        }
        *(float4*)&sums[grp][piece >> 5][((piece & 31) >> 2) * LS + 4 * (piece & 3)] = s;
        ahead(ch + nbg < nchunks ? t : t - 1, ch + nbg < nchunks ? ch + nbg : bgrp);
        if (!__syncthreads_and(ok ? 1 : 0)) {
          if (threadIdx.x == 0) atomicCAS(dev_err, 0, 3003);
          return;
        }
        if (ring < T && t % MQ_FENCE == 0) __threadfence();
        if (mine) {
          float r = 0.0f;
#pragma unroll
          for (int w = 0; w < GRP; ++w) r += sums[w][gb >> 3][(gu & 7) * LS + 4 * ((gb & 7) >> 1) + (gb & 1) + 2 * (gu >> 3)];
          dh += r;
        }
      } else {
        ahead(ch + nbg < nchunks ? t : t - 1, ch + nbg < nchunks ? ch + nbg : bgrp);
        if (ci > 0) __syncthreads();   // (no poll, so no barrier yet: the chunk before may still be read from frag, csh and dval)
      }
      float d[NG];
#pragma unroll
      for (int g = 0; g < NG; ++g) d[g] = 0.0f;
      if (mine) {
        float* cy = carry + ci * BLOCK + threadIdx.x;
        if (NG == 4) {
          const float tc = tanhf(ct);
          const float d_o = dh * tc;
          const float dcc = *cy + dh * k3 * (1.0f - tc * tc);
          d[0] = dcc * k2 * k0 * (1.0f - k0);
          d[1] = dcc * sp * k1 * (1.0f - k1);
          d[2] = dcc * k0 * (1.0f - k2 * k2);
          d[NG - 1] = d_o * k3 * (1.0f - k3);
          *cy = dcc * k1;
        } else {
          if (t < T - 1) dh += *cy;
          const float r = k0, z = k1, hc = k2, gh3 = k3;
          const float da3 = dh * (1.0f - z) * (1.0f - hc * hc);
          const float da2 = dh * (sp - hc) * z * (1.0f - z);
          const float da1 = da3 * gh3 * r * (1.0f - r);
          d[0] = da1; d[1] = da2; d[2] = da3 * r;
          float* x = dgx + (int64_t)t * K + (int64_t)b * ldd;
          x[u] = da1; x[H + u] = da2; x[2 * H + u] = da3;
          *cy = dh * z;
        }
      }
      if (t > 0 && gates) {
        // this column's planes (zeros for units and columns that do not exist), scaled by its largest value
        uint32_t m = 0u;
#pragma unroll
        for (int g = 0; g < NG; ++g) m = max(m, __float_as_uint(d[g]) & 0x7fffffffu);
#pragma unroll
        for (int o = 1; o < UG; o *= 2) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
        const int sh = mq_shift(m);
        const float sc = mq_pow2(sh);
        if (gu == 0) csh[gb] = m < MQ_INF ? sh : MQ_BAD;
#pragma unroll
        for (int g = 0; g < NG; ++g) {
          const float x = d[g] * sc;
          const __half hi = __float2half_rn(x), lo = __float2half_rn(x - __half2float(hi));
          __half* f = (__half*)&frag[g][gb >> 3][4 * (gb & 7) + (gu >> 2)] + (gu & 3);
          f[0] = hi;
          f[4] = lo;
          dval[gb][g * UG + gu] = d[g];
        }
      }
      __syncthreads();   // planes are there for all; in step 0 nothing is, but the next chunk's partial sums go where these have been read
      if (mine) {
        float* row = dg + (int64_t)t * K + (int64_t)b * ldd;
#pragma unroll
        for (int g = 0; g < NG; ++g) row[g * H + u] = d[g];
      }
      if (t == 0) continue;
      uint4 bf[NG][NT];
      int sh[NT][2];
      bool cols = true;
#pragma unroll
      for (int n = 0; n < NT; ++n) {
#pragma unroll
        for (int g = 0; g < NG; ++g) bf[g][n] = frag[g][n][lane];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          sh[n][i] = csh[8 * n + 2 * q + i];
          cols = cols && sh[n][i] != MQ_BAD;
        }
      }
      float* dst = ex + (size_t)(t % ring) * run + ((size_t)ch * ugroups * ugroups + ug) * BLOCK + 4 * lane;
      auto send = [&](int m, int n, const float (&v)[4]) {
        if (warp + 8 * m < ugroups) mq_put4(dst + (size_t)(warp + 8 * m) * ugroups * BLOCK + 128 * n, mq_word(v[0]), mq_word(v[1]), mq_word(v[2]), mq_word(v[3]));
      };
      // (groups that do not exist have rows of zeros: no branch between the products, so that one group's sums are scaled and sent under
      // the next one's products)
      auto products = [&](auto is_plain) {
        float f[NT][2];
#pragma unroll
        for (int n = 0; n < NT; ++n)
#pragma unroll
          for (int i = 0; i < 2; ++i) f[n][i] = mq_pow2(-sh[n][i]);
#pragma unroll
        for (int m = 0; m < MT; ++m) {
          constexpr int CR = MT < 4 ? 2 : 1;   // (four groups leave no registers for more)
          float hh[NT][4], cr[CR][NT][4];      // hi hi, and the cross terms: sums of their own, as an mma waits for the one that it adds to
#pragma unroll
          for (int n = 0; n < NT; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) hh[n][e] = cr[0][n][e] = cr[CR - 1][n][e] = 0.0f;
#pragma unroll
          for (int g = 0; g < NG; ++g) {
#pragma unroll
            for (int n = 0; n < NT; ++n) mq_mma(cr[0][n], alo[m][g], bf[g][n].x, bf[g][n].y);
#pragma unroll
            for (int n = 0; n < NT; ++n) mq_mma(hh[n], ahi[m][g], bf[g][n].x, bf[g][n].y);
#pragma unroll
            for (int n = 0; n < NT; ++n) mq_mma(cr[CR - 1][n], ahi[m][g], bf[g][n].z, bf[g][n].w);
          }
          const float a0 = mq_pow2(-ash[m][0]), a1 = mq_pow2(-ash[m][1]);
#pragma unroll
          for (int n = 0; n < NT; ++n) {
            float v[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const float x = CR == 2 ? hh[n][e] + (cr[0][n][e] + cr[CR - 1][n][e]) : hh[n][e] + cr[0][n][e];
              v[e] = decltype(is_plain)::value ? x * ((e >> 1 ? a1 : a0) * f[n][e & 1]) : mq_unscale(x, -(ash[m][e >> 1] + sh[n][e & 1]));
            }
            send(m, n, v);
          }
        }
      };
      bool plain = moderate;
#pragma unroll
      for (int n = 0; n < NT; ++n) plain = plain && abs(sh[n][0]) <= MQ_MODERATE && abs(sh[n][1]) <= MQ_MODERATE;
      plain = __all_sync(0xffffffffu, plain);
      if (__all_sync(0xffffffffu, cols && finite)) {
        if (plain) products(std::true_type());
        else products(std::false_type());
      } else {
        for (int m = 0; m < MT; ++m) {
          float v[NT][4];
#pragma unroll
          for (int n = 0; n < NT; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) v[n][e] = 0.0f;
          for (int k = 0; k < NG * UG; ++k) {
            const int g = k / UG, w = u0 + k % UG;
            if (w >= H) continue;
#pragma unroll
            for (int n = 0; n < NT; ++n)
#pragma unroll
              for (int e = 0; e < 4; ++e) {
                const int c = 8 * n + 2 * q + (e & 1), row = (warp + 8 * m) * UG + (lane >> 2) + 8 * (e >> 1);
                if (c < nb && row < H) v[n][e] = fmaf(__ldg(Wh + (int64_t)row * K + g * H + w), dval[c][k], v[n][e]);
              }
          }
#pragma unroll
          for (int n = 0; n < NT; ++n) send(m, n, v[n]);
        }
      }
    }
  }
}
