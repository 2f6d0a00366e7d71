// The whole time loop of an LSTM / GRU in one launch, any hidden size that fits and any batch (included by recurrent.cu).
//
// Forward.  CTA (unit group, batch group) owns UG hidden units - their NG * UG gate rows of Wh stay in shared memory for all
// T steps - and walks BG batch columns at a time (several chunks when the batch is larger than the grid).  A step needs
// h_{t-1} of its columns from every unit group.
//
// What bounds it: T dependent steps, each one exchange of h through L2 plus the FMAs of the CTA's rows (UG 16, BG 16,
// H 512: 4096 cycles at full rate).  A barrier between steps (atomic arrival, poll, then the loads) costs three L2 round
// trips; here the data are their own flag: `out` is filled with a NaN pattern no result has (0xffffffff) before the launch,
// a step's stores are 4-byte relaxed stores, and a consumer polls the very words it needs until none of them is the
// pattern: one store -> load flight per step, no fence, no barrier, no counter.  Every word is written once per launch, so
// there is nothing to reset and no slot to reuse.  A NaN result with that pattern is stored as 0x7fffffff.
//
// The product: 256 threads = 8 warps that share k (a warp takes one eighth of it), a lane owns NG * UG / 8 rows x BG / 4
// columns, both operands K-major with padded rows, read by 128-bit loads (12 loads per 128 FMAs at 64 x 16; the 4 x 4
// tiles of an earlier kernel needed 8 per 64 and were bound by the shared-memory pipe: such a load takes 2 cycles of it when
// every 8 lanes name at most 2 addresses, else 4).  Partial sums of the warps meet
// in shared memory where thread (unit, column) applies the gates.
//
// Backward.  The same CTA computes dh_t of its units: the derivatives dg_{t+1} of all NG * H gate rows of its columns
// (polled in pieces of 512 rows, the next piece in flight while one is multiplied) times its UG rows of Wh' (resident),
// then turns dh into its own gate derivatives dg_t.  One exchange per step, no partial sums in memory.
//
// Polls are bounded: code 3002 (forward) / 3003 (backward) lands in the device error word and every CTA leaves its loop.
#pragma once

constexpr int SQ_THREADS = 256, SQ_KC = 512;
constexpr uint32_t SQ_EMPTY = 0xffffffffu;
constexpr uint32_t SQ_POLL_LIMIT = 1u << 21;

__device__ __forceinline__ void sq_publish(float* p, float v) {
  uint32_t u = __float_as_uint(v);
  if (u == SQ_EMPTY) u = 0x7fffffffu;
  asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(u) : "memory");
}
__device__ __forceinline__ uint4 sq_peek4(const float* p) {
  uint4 v;
  asm volatile("ld.relaxed.gpu.global.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ uint32_t sq_peek(const float* p) {
  uint32_t v;
  asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// acc.{even k, odd k} += w * h for four k values: packed FMAs take two k values per instruction straight from K-major
// operands (measured on B200: 3.7 FMAs per cycle and SM partition set against 3.0 for single ones, at half the issue slots)
__device__ __forceinline__ void sq_fma4(unsigned long long& acc, const ulonglong2& w, const ulonglong2& h) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(w.x), "l"(h.x));
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(w.y), "l"(h.y));
}
__device__ __forceinline__ float sq_sum2(unsigned long long acc) {
  return __uint_as_float((uint32_t)acc) + __uint_as_float((uint32_t)(acc >> 32));
}

// Values [c0, c0 + 32 * PER) of the rows warp, warp + 8, ... (RW of them) of a [rows][cols] array whose rows are ld apart,
// as float4s (PER / 4 per lane and row) or single words, polled until present (poll) or read once.  v holds them in
// registers; sq_store puts them into shared memory.
template <int RW, int PER>
struct SqPiece {
  uint32_t v[RW][PER];
  template <bool VEC>
  __device__ __forceinline__ bool fetch(const float* src, int64_t ld, int nrows, int c0, int cols, bool poll, const int32_t* dev_err) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    bool ok = true;
    uint32_t spins = 0;
    for (;;) {
      bool missing = false;
#pragma unroll
      for (int r = 0; r < RW; ++r) {
        const int row = warp + 8 * r;
        const float* p = src + (int64_t)row * ld;
        if (VEC) {
#pragma unroll
          for (int q = 0; q < PER / 4; ++q) {
            const int c = c0 + 4 * (lane + 32 * q);
            uint4 x = make_uint4(0u, 0u, 0u, 0u);
            if (row < nrows && c < cols) x = sq_peek4(p + c);
            missing |= (x.x == SQ_EMPTY) | (x.y == SQ_EMPTY) | (x.z == SQ_EMPTY) | (x.w == SQ_EMPTY);
            v[r][4 * q] = x.x; v[r][4 * q + 1] = x.y; v[r][4 * q + 2] = x.z; v[r][4 * q + 3] = x.w;
          }
        } else {
#pragma unroll
          for (int q = 0; q < PER; ++q) {
            const int c = c0 + lane + 32 * q;
            uint32_t x = 0u;
            if (row < nrows && c < cols) x = sq_peek(p + c);
            missing |= (x == SQ_EMPTY);
            v[r][q] = x;
          }
        }
      }
      if (!poll || !missing) break;
      if (++spins > SQ_POLL_LIMIT || ((spins & 255u) == 255u && *(const volatile int32_t*)dev_err != 0)) { ok = false; break; }
    }
    return ok;
  }
  __device__ __forceinline__ bool complete() const {
    bool missing = false;
#pragma unroll
    for (int r = 0; r < RW; ++r)
#pragma unroll
      for (int q = 0; q < PER; ++q) missing |= v[r][q] == SQ_EMPTY;
    return !missing;
  }
  // columns below lim (relative to c0); what lies beyond the array was read as zeros
  template <bool VEC>
  __device__ __forceinline__ void store(float* dst, int lds, int nrows, int lim) const {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
    for (int r = 0; r < RW; ++r) {
      const int row = warp + 8 * r;
      if (row >= nrows) continue;
      if (VEC) {
#pragma unroll
        for (int q = 0; q < PER / 4; ++q) {
          const int c = 4 * (lane + 32 * q);
          if (c < lim) *(uint4*)(dst + row * lds + c) = make_uint4(v[r][4 * q], v[r][4 * q + 1], v[r][4 * q + 2], v[r][4 * q + 3]);
        }
      } else {
#pragma unroll
        for (int q = 0; q < PER; ++q) {
          const int c = lane + 32 * q;
          if (c < lim) dst[row * lds + c] = __uint_as_float(v[r][q]);
        }
      }
    }
  }
};

inline int sq_pad(int n, int m) { return (n + m - 1) / m * m; }
inline size_t sq_fwd_smem(int ng, int ug, int bg, int H, int chunks) {
  const int ld = sq_pad(H, 32) + 4;
  return ((size_t)ng * ug * ld + (size_t)bg * ld + (size_t)8 * ng * ug * (bg + 1) + (size_t)chunks * ug * bg) * 4;
}
inline size_t sq_bwd_smem(int ng, int ug, int bg, int H, int chunks) {
  const size_t piece = (size_t)bg * (SQ_KC + 16), sums = (size_t)32 * (ug * bg + 2);
  return ((size_t)ug * (sq_pad(ng * H, SQ_KC) + 16) + 2 * (piece > sums ? piece : sums) + (size_t)chunks * ug * bg) * 4;
}

// LSTM (NG = 4): cache = gates [rows][4H] or NULL, cst = cell states ([rows][H] when cached), gx [rows][4H].
// GRU (NG = 3): cache = (r, z, hc, gh3) [rows][4H] or NULL, gx [rows][3H]; c0 / cst / cT unused.
template <int NG, int UG, int BG, bool VEC>
__global__ void __launch_bounds__(SQ_THREADS, 1)
rnn_fwd_seq_kernel(const float* __restrict__ Wh, const float* __restrict__ gx, const float* __restrict__ h0, const float* __restrict__ c0,
                   float* out, float* cache, float* cst, int cached, float* __restrict__ hT, float* __restrict__ cT, int H, int B, int T,
                   int nbg, int32_t* dev_err) {
  constexpr int R = NG * UG, TR = R / 8, TC = BG / 4, RW = BG >= 8 ? BG / 8 : 1;
  extern __shared__ __align__(16) float sm[];
  const int Hp = (H + 31) & ~31, ld = Hp + 4;
  float* Ws = sm;                            // [R][ld]
  float* hs = Ws + (size_t)R * ld;           // [BG][ld]
  float* red = hs + (size_t)BG * ld;         // [8][R][BG + 1]
  float* cs = red + 8 * R * (BG + 1);        // [chunks][UG * BG]
  const int ugroups = (H + UG - 1) / UG;
  const int u0 = ((int)blockIdx.x % ugroups) * UG, bgrp = (int)blockIdx.x / ugroups;
  const int nchunks = (B + BG - 1) / BG;
  const int64_t ldrow = (int64_t)T * H, ldgx = (int64_t)T * NG * H, ldc = (int64_t)T * 4 * H;
  for (int e = threadIdx.x; e < BG * ld; e += SQ_THREADS) hs[e] = 0.0f;
  // Ws[g * UG + u][k] = Wh[g * H + u0 + u][k] from the weight memory [H (k)][NG * H]
  for (int e = threadIdx.x; e < R * Hp; e += SQ_THREADS) {
    const int rr = e % R, k = e / R, g = rr / UG, u = rr % UG;
    Ws[(size_t)rr * ld + k] = (k < H && u0 + u < H) ? __ldg(Wh + (int64_t)k * (NG * H) + g * H + u0 + u) : 0.0f;
  }
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rg = lane >> 2, cg = lane & 3;          // product: rows rg + 8 i, columns cg + 4 j
  const int gu = threadIdx.x % UG, gb = threadIdx.x / UG;   // gates: unit, column (threads below UG * BG)
  const int u = u0 + gu;
  if (NG == 4)
    for (int ch = bgrp, i = 0; ch < nchunks; ch += nbg, ++i) {
      const int b = ch * BG + gb;
      if (threadIdx.x < UG * BG) cs[i * UG * BG + threadIdx.x] = (c0 && b < B && u < H) ? c0[(int64_t)b * H + u] : 0.0f;
    }
  __syncthreads();
  const int kper = Hp >> 3;
  SqPiece<RW, 16> pc;
  bool fetched = false;
  for (int t = 0; t < T; ++t) {
    const float* hprev = t == 0 ? h0 : out + (int64_t)(t - 1) * H;
    const int64_t ldh = t == 0 ? H : ldrow;
    for (int ch = bgrp, ci = 0; ch < nchunks; ch += nbg, ++ci) {
      const int b0 = ch * BG, nb = B - b0 < BG ? B - b0 : BG;
      const int b = b0 + gb;
      const bool mine = threadIdx.x < UG * BG && gb < nb && u < H;
      float gxv[NG];
#pragma unroll
      for (int g = 0; g < NG; ++g) gxv[g] = mine ? __ldg(gx + (int64_t)b * ldgx + (int64_t)t * NG * H + g * H + u) : 0.0f;
      unsigned long long acc[TR][TC];
#pragma unroll
      for (int i = 0; i < TR; ++i)
#pragma unroll
        for (int j = 0; j < TC; ++j) acc[i][j] = 0ull;
      if (hprev != nullptr) {
        int ok = 1;
        const float* src = hprev + (int64_t)b0 * ldh;
        for (int c = 0; c < H; c += SQ_KC) {
          if (!fetched || c > 0 || !pc.complete()) ok &= pc.template fetch<VEC>(src, ldh, nb, c, H, t > 0, dev_err) ? 1 : 0;
          pc.template store<VEC>(hs + c, ld, nb, H - c);
        }
        if (!__syncthreads_and(ok)) {
          if (threadIdx.x == 0) atomicCAS(dev_err, 0, 3002);
          return;
        }
        // several chunks: the first columns of the next one are on their way while this one is multiplied
        fetched = ch + nbg < nchunks;
        if (fetched) pc.template fetch<VEC>(src + (int64_t)nbg * BG * ldh, ldh, B - b0 - nbg * BG < BG ? B - b0 - nbg * BG : BG, 0, H, false, dev_err);
        const float* wp = Ws + (size_t)rg * ld + warp * kper;
        const float* hp = hs + cg * ld + warp * kper;
#pragma unroll 4
        for (int k = 0; k < kper; k += 4) {
          ulonglong2 w[TR], h[TC];
#pragma unroll
          for (int j = 0; j < TC; ++j) h[j] = *(const ulonglong2*)(hp + 4 * j * ld + k);
#pragma unroll
          for (int i = 0; i < TR; ++i) w[i] = *(const ulonglong2*)(wp + (size_t)(8 * i) * ld + k);
#pragma unroll
          for (int i = 0; i < TR; ++i)
#pragma unroll
            for (int j = 0; j < TC; ++j) sq_fma4(acc[i][j], w[i], h[j]);
        }
      }
      if (hprev == nullptr) __syncthreads();   // (the other path has passed one) red of the previous chunk has been read
      float hp_own = 0.0f;
      if (NG == 3 && hprev != nullptr && mine) hp_own = hs[gb * ld + u];   // before the barrier: hs is refilled after it
#pragma unroll
      for (int i = 0; i < TR; ++i)
#pragma unroll
        for (int j = 0; j < TC; ++j) red[(warp * R + rg + 8 * i) * (BG + 1) + cg + 4 * j] = sq_sum2(acc[i][j]);
      __syncthreads();
      if (mine) {
        float pre[NG];
#pragma unroll
        for (int g = 0; g < NG; ++g) {
          float s = 0.0f;
#pragma unroll
          for (int w = 0; w < 8; ++w) s += red[(w * R + g * UG + gu) * (BG + 1) + gb];
          pre[g] = s;
        }
        float hn, cn = 0.0f;
        float4 keep;
        if (NG == 4) {
          const float zi = pre[0] + gxv[0], zf = pre[1] + gxv[1], zg = pre[2] + gxv[2], zo = pre[NG - 1] + gxv[NG - 1];
          const float ig = 1.0f / (1.0f + expf(-zi)), fg = 1.0f / (1.0f + expf(-zf));
          const float gg = tanhf(zg), og = 1.0f / (1.0f + expf(-zo));
          float* c = cs + ci * UG * BG + threadIdx.x;
          cn = fg * *c + ig * gg;
          *c = cn;
          hn = og * tanhf(cn);
          keep = make_float4(ig, fg, gg, og);
        } else {
          const float gh3 = pre[2];
          const float r = 1.0f / (1.0f + expf(-(gxv[0] + pre[0])));
          const float z = 1.0f / (1.0f + expf(-(gxv[1] + pre[1])));
          const float hc = tanhf(gxv[2] + r * gh3);
          hn = (1.0f - z) * hc + z * hp_own;
          keep = make_float4(r, z, hc, gh3);
        }
        sq_publish(out + (int64_t)t * H + (int64_t)b * ldrow + u, hn);
        if (cache) {
          float* gr = cache + (int64_t)t * 4 * H + (int64_t)b * ldc;
          gr[u] = keep.x; gr[H + u] = keep.y; gr[2 * H + u] = keep.z; gr[3 * H + u] = keep.w;
        }
        if (NG == 4 && cached) cst[(int64_t)t * H + (int64_t)b * ldrow + u] = cn;
        if (t == T - 1 && hT) {
          hT[(int64_t)b * H + u] = hn;
          if (NG == 4) cT[(int64_t)b * H + u] = cn;
        }
      }
    }
  }
}

// LSTM: keep = gates [rows][4H] (read), cst = cell states, dg [rows][4H] = gate derivatives (filled with the pattern before the
// launch).  GRU: keep = (r, z, hc, gh3) [rows][4H], hout = the forward output, dg = recurrent-side derivatives [rows][3H]
// (filled with the pattern), dgx = input-side derivatives [rows][3H].
template <int NG, int UG, int BG, bool VEC>
__global__ void __launch_bounds__(SQ_THREADS, 1)
rnn_bwd_seq_kernel(const float* __restrict__ Wh, const float* __restrict__ keep, const float* __restrict__ cst,
                   const float* __restrict__ s0, const float* __restrict__ hout, const float* __restrict__ dout,
                   const float* __restrict__ dhT, const float* __restrict__ dcT, float* dg, float* __restrict__ dgx, int H, int B, int T,
                   int nbg, int32_t* dev_err) {
  constexpr int TR = UG / 2, TC = BG / 4, RW = BG >= 8 ? BG / 8 : 1;
  extern __shared__ __align__(16) float sm[];
  const int K = NG * H, Kp = (K + SQ_KC - 1) / SQ_KC * SQ_KC, ldw = Kp + 16;
  constexpr int LDD = SQ_KC + 16;
  float* Ws = sm;                                 // [UG][ldw]
  constexpr int BUF = BG * LDD > 32 * (UG * BG + 2) ? BG * LDD : 32 * (UG * BG + 2);
  float* Ds = Ws + (size_t)UG * ldw;              // two of [BG][LDD]; [32][UG * BG + 2] for the reduction
  float* carry = Ds + 2 * BUF;                    // [chunks][UG * BG]: LSTM dc, GRU dh * z
  const int ugroups = (H + UG - 1) / UG;
  const int u0 = ((int)blockIdx.x % ugroups) * UG, bgrp = (int)blockIdx.x / ugroups;
  const int nchunks = (B + BG - 1) / BG;
  const int64_t ldrow = (int64_t)T * H, ldd = (int64_t)T * K, ldk = (int64_t)T * 4 * H;
  for (int e = threadIdx.x; e < 2 * BUF; e += SQ_THREADS) Ds[e] = 0.0f;
  for (int e = threadIdx.x; e < UG * Kp; e += SQ_THREADS) {
    const int r = e % Kp, uu = e / Kp;
    Ws[(size_t)uu * ldw + r] = (r < K && u0 + uu < H) ? __ldg(Wh + (int64_t)(u0 + uu) * K + r) : 0.0f;
  }
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int pu = lane & 1, pc = (lane >> 1) & 3, kg = warp * 4 + (lane >> 3);   // product: units pu + 2 i, columns pc + 4 j, k group
  const int gu = threadIdx.x % UG, gb = threadIdx.x / UG;
  const int u = u0 + gu;
  SqPiece<RW, 16> piece;
  bool fetched = false;
  float* buf = Ds;
  for (int ch = bgrp, i = 0; ch < nchunks; ch += nbg, ++i) {
    const int b = ch * BG + gb;
    if (threadIdx.x < UG * BG) carry[i * UG * BG + threadIdx.x] = (NG == 4 && dcT && b < B && u < H) ? dcT[(int64_t)b * H + u] : 0.0f;
  }
  __syncthreads();
  for (int t = T - 1; t >= 0; --t) {
    for (int ch = bgrp, ci = 0; ch < nchunks; ch += nbg, ++ci) {
      const int b0 = ch * BG, nb = B - b0 < BG ? B - b0 : BG;
      const int b = b0 + gb;
      const bool mine = threadIdx.x < UG * BG && gb < nb && u < H;
      float k0 = 0.f, k1 = 0.f, k2 = 0.f, k3 = 0.f, ct = 0.f, sp = 0.f, dh = 0.f;
      if (mine) {
        const float* kr = keep + (int64_t)t * 4 * H + (int64_t)b * ldk;
        k0 = __ldg(kr + u); k1 = __ldg(kr + H + u); k2 = __ldg(kr + 2 * H + u); k3 = __ldg(kr + 3 * H + u);
        const float* prev = NG == 4 ? cst : hout;   // c_{t-1} or h_{t-1}
        if (NG == 4) ct = __ldg(cst + (int64_t)t * H + (int64_t)b * ldrow + u);
        sp = t > 0 ? __ldg(prev + (int64_t)(t - 1) * H + (int64_t)b * ldrow + u) : s0 ? __ldg(s0 + (int64_t)b * H + u) : 0.0f;
        dh = __ldg(dout + (int64_t)t * H + (int64_t)b * ldrow + u);
        if (t == T - 1 && dhT) dh += __ldg(dhT + (int64_t)b * H + u);
      }
      if (t < T - 1) {
        const float* src = dg + (int64_t)(t + 1) * K + (int64_t)b0 * ldd;
        unsigned long long acc[TR][TC];
#pragma unroll
        for (int i = 0; i < TR; ++i)
#pragma unroll
          for (int j = 0; j < TC; ++j) acc[i][j] = 0ull;
        int ok = (fetched && piece.complete()) || piece.template fetch<VEC>(src, ldd, nb, 0, K, true, dev_err) ? 1 : 0;
        fetched = false;
        for (int c = 0; c < K; c += SQ_KC, buf = buf == Ds ? Ds + BUF : Ds) {
          piece.template store<VEC>(buf, LDD, nb, SQ_KC);   // (every thread is past the product of the piece before last)
          if (!__syncthreads_and(ok)) {
            if (threadIdx.x == 0) atomicCAS(dev_err, 0, 3003);
            return;
          }
          // the next piece (or the next chunk's first) is on its way while this one is multiplied; it is looked at again
          // only if it was not complete
          const bool more = c + SQ_KC < K;
          if (more) piece.template fetch<VEC>(src, ldd, nb, c + SQ_KC, K, false, dev_err);
          else if (ch + nbg < nchunks) {
            fetched = true;
            piece.template fetch<VEC>(src + (int64_t)nbg * BG * ldd, ldd, B - b0 - nbg * BG < BG ? B - b0 - nbg * BG : BG, 0, K, false, dev_err);
          }
          const float* wp = Ws + (size_t)pu * ldw + c + 4 * kg;
          const float* dp = buf + pc * LDD + 4 * kg;
          const int lim = K - c < SQ_KC ? K - c : SQ_KC;
#pragma unroll 4
          for (int k = 0; k < lim; k += 128) {
            ulonglong2 w[TR], d[TC];
#pragma unroll
            for (int j = 0; j < TC; ++j) d[j] = *(const ulonglong2*)(dp + 4 * j * LDD + k);
#pragma unroll
            for (int i = 0; i < TR; ++i) w[i] = *(const ulonglong2*)(wp + (size_t)(2 * i) * ldw + k);
#pragma unroll
            for (int i = 0; i < TR; ++i)
#pragma unroll
              for (int j = 0; j < TC; ++j) sq_fma4(acc[i][j], w[i], d[j]);
          }
          if (more) ok = piece.complete() || piece.template fetch<VEC>(src, ldd, nb, c + SQ_KC, K, true, dev_err) ? 1 : 0;
        }
        // the k groups' sums go where the piece before the last was (buf points there)
        float* red = buf;
        buf = buf == Ds ? Ds + BUF : Ds;   // the next piece must not overwrite sums that are still being read
#pragma unroll
        for (int i = 0; i < TR; ++i)
#pragma unroll
          for (int j = 0; j < TC; ++j) red[kg * (UG * BG + 2) + (pc + 4 * j) * UG + pu + 2 * i] = sq_sum2(acc[i][j]);
        __syncthreads();
        if (mine) {
          float s = 0.0f;
#pragma unroll 8
          for (int g = 0; g < 32; ++g) s += red[g * (UG * BG + 2) + gb * UG + gu];
          dh += s;
        }
      }
      if (mine) {
        float* cy = carry + ci * UG * BG + threadIdx.x;
        float* row = dg + (int64_t)t * K + (int64_t)b * ldd;
        if (NG == 4) {
          const float tc = tanhf(ct);
          const float d_o = dh * tc;
          const float dcc = *cy + dh * k3 * (1.0f - tc * tc);
          sq_publish(row + u, dcc * k2 * k0 * (1.0f - k0));
          sq_publish(row + H + u, dcc * sp * k1 * (1.0f - k1));
          sq_publish(row + 2 * H + u, dcc * k0 * (1.0f - k2 * k2));
          sq_publish(row + 3 * H + u, d_o * k3 * (1.0f - k3));
          *cy = dcc * k1;
        } else {
          if (t < T - 1) dh += *cy;
          const float r = k0, z = k1, hc = k2, gh3 = k3;
          const float da3 = dh * (1.0f - z) * (1.0f - hc * hc);
          const float da2 = dh * (sp - hc) * z * (1.0f - z);
          const float da1 = da3 * gh3 * r * (1.0f - r);
          sq_publish(row + u, da1);
          sq_publish(row + H + u, da2);
          sq_publish(row + 2 * H + u, da3 * r);
          float* x = dgx + (int64_t)t * K + (int64_t)b * ldd;
          x[u] = da1; x[H + u] = da2; x[2 * H + u] = da3;
          *cy = dh * z;
        }
      }
    }
  }
}
