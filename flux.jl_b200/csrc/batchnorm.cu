// BatchNorm forward (training / inference) and backward (memory-bound).
//
// Data layout: x is [n][c][s] row-major (Julia WHCN with s = W*H; a 2-D input [C, N] has s == 1).  A block of 256 threads takes
// rows (one sample's s values of a channel) with tpr threads side by side on one row (a power of two) and 256 / tpr rows at a
// time; W = 4 floats a piece where rows are whole aligned float4, else one.
//
// Training forward: a cluster of up to 8 CTAs owns a channel at a time.  Its values are read once, into shared memory, where their
// statistics are taken; the CTAs' sums meet in distributed shared memory, and y is written from there: 1 read + 1 write.  The
// kernel is persistent: while a channel is worked on the next two are on their way.  Channels that do not fit
// (more than 8 x 200 KB) take statistics first and normalise in a second pass.  32 x 32 x 256 x 128: 76 -> 63 us (statistics, a
// finaliser and a second pass before; 41 would be two passes at the HBM rate: 15 clusters of 8 fit the GPU, 120 of 148 SMs,
// and 256 channels are 17.1 rounds of them); 7 x 7 x 512 x 256: 136 -> 21; 512 x 256: 103 -> 7.
// Backward: sums of dz and dz xhat per channel (a cluster again, no second launch), then, if dx is wanted, a pass that writes
// it; the activation mask is recomputed from x instead of reading y.
// Statistics: a thread adds x - shift and its square with the first of its own values as the shift, over at most a few hundred values;
// count, mean and sum of squared deviations of threads, warps and CTAs are then merged (Chan, Golub and LeVeque, "Updating formulae
// and a pairwise algorithm for computing sample variances").  So nothing cancels when |mean| / std is large, wherever the channel's
// first value lies: mean / std = 1000 and a first value of 0, 131072 values: variance off by 3e-5 (as sums over the channel: 1e-2).
#include "common.cuh"
#include "tc_common.cuh"

namespace {

constexpr int BN_THREADS = 256;
constexpr int BN_FWD_THREADS = 512;          // of a channel cached in shared memory: more loads of one CTA in flight
constexpr int BN_MAX_CLUSTER = 8;
constexpr size_t BN_CACHE_MAX = 200 * 1024;  // of one CTA, the only one of its SM

template <int W>
__device__ __forceinline__ void ld_piece(const float* p, float* v) {
  if (W == 4) {
    const float4 q = *(const float4*)p;
    v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
  } else {
    v[0] = *p;
  }
}
// the same for values that are not looked at again soon (whole passes over tensors that may exceed L2)
template <int W>
__device__ __forceinline__ void ld_stream(const float* p, float* v) {
  if (W == 4) {
    const float4 q = __ldcs((const float4*)p);
    v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
  } else {
    v[0] = *p;
  }
}
template <int W>
__device__ __forceinline__ void st_stream(float* p, const float* v) {
  if (W == 4) __stcs((float4*)p, make_float4(v[0], v[1], v[2], v[3]));
  else *p = v[0];
}
template <int W>
__device__ __forceinline__ void st_piece(float* p, const float* v) {
  if (W == 4) *(float4*)p = make_float4(v[0], v[1], v[2], v[3]);
  else *p = v[0];
}

struct Dims {
  int64_t s, c, n;
  int split;   // CTAs per channel
  int tpr;     // threads side by side on one row
};

// The pieces of a channel that this thread owns: `mine` rows, `step` floats apart, in each of `cols` columns of pieces, `col_step`
// floats apart, the first of channel 0 at `base`.
struct Walk {
  int64_t base, step;
  int mine, cols, col_step;
};
template <int W>
__device__ __forceinline__ Walk make_walk(const Dims& g, int p) {
  const int tx = threadIdx.x & (g.tpr - 1), ty = threadIdx.x / g.tpr, nr = (int)blockDim.x / g.tpr;
  const int64_t first = (int64_t)p * nr + ty, rows = (int64_t)g.split * nr, mine = (g.n - first + rows - 1) / rows;
  const int64_t at = (int64_t)tx * W, cols = (g.s - at + (int64_t)g.tpr * W - 1) / ((int64_t)g.tpr * W);
  Walk w;
  w.base = first * g.c * g.s + at;
  w.step = rows * g.c * g.s;
  w.mine = first < g.n ? (int)mine : 0;
  w.cols = at < g.s ? (int)cols : 0;
  w.col_step = g.tpr * W;
  return w;
}
// f(k, off, m), U rows at a time, in an order that a second call repeats: pieces k .. k + m - 1 (m <= U) of channel ch lie at off,
// off + w.step, ...
template <int U, typename F>
__device__ __forceinline__ void each_piece(const Walk& w, int64_t ch_off, F f) {
  int k = 0;
  for (int j = 0; j < w.cols; ++j) {
    int64_t off = w.base + ch_off + (int64_t)j * w.col_step;
    for (int i = 0; i < w.mine; i += U, off += U * w.step) {
      const int m = w.mine - i < U ? w.mine - i : U;
      f(k, off, m);
      k += m;
    }
  }
}

// Values of the CTAs of a cluster of `split`.  Every CTA sends its own to all of them with st.async, which an mbarrier of the receiver
// counts: a cluster barrier would first wait for every store to y that is still on its way (its release covers them): that cost
// 1 - 2 us of the 5 us a channel of 32 x 32 x 128 values took.  Two sets of slots in turn: a CTA sends to a set again only after
// everybody's next values have reached it, which are sent after this set was read.
struct Exchange {
  float4 slots[2][BN_MAX_CLUSTER];
  uint64_t bar[2];
  float sh[64];
  float warp_n[32];   // values of each warp
};
__device__ __forceinline__ void exchange_init(Exchange& x, int split) {
  if (split == 1) return;
  if (threadIdx.x == 0) {
    mbar_init(smem_u32(&x.bar[0]), 1);
    mbar_init(smem_u32(&x.bar[1]), 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncwarp();
  cluster_sync_all();
}
// One warp sends the CTA's values (the same in each of its lanes).
__device__ __forceinline__ void exchange_send(Exchange& x, const float4& v, int split, uint32_t mine, int round) {
  const int lane = threadIdx.x & 31, turn = round & 1;
  const uint32_t bar = smem_u32(&x.bar[turn]);
  if (lane == 0) mbar_arrive_expect_tx(bar, 16u * (uint32_t)split);
  if (lane < split)
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.f32 [%0], {%1, %2, %3, %4}, [%5];"
                 ::"r"(map_to_cta(smem_u32(&x.slots[turn][mine]), (uint32_t)lane)), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w),
                 "r"(map_to_cta(bar, (uint32_t)lane))
                 : "memory");
}
// Waits for everybody's values of this round (`round` counts the calls); false when the wait ran out (bounded: error code 2101).
__device__ __forceinline__ bool exchange_wait(Exchange& x, int round) {
  uint32_t ok = 0;
  for (uint32_t it = 0; it < WAIT_LIMIT && !ok; ++it)
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(&x.bar[round & 1])), "r"((uint32_t)(round >> 1) & 1u)
        : "memory");
  return ok != 0;
}

// Both sums over the cluster, valid in every thread.
__device__ __forceinline__ bool channel_sums(Exchange& x, float& a, float& b, int split, uint32_t mine, int round) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = (int)blockDim.x >> 5;
  a = fb_warp_sum(a);
  b = fb_warp_sum(b);
  if (lane == 0) { x.sh[w] = a; x.sh[32 + w] = b; }
  __syncthreads();
  if (split == 1 || w == 0) {
    a = fb_warp_sum(lane < nw ? x.sh[lane] : 0.0f);
    b = fb_warp_sum(lane < nw ? x.sh[32 + lane] : 0.0f);
  }
  if (split == 1) {
    __syncthreads();   // sh may be written again
    return true;
  }
  if (w == 0) exchange_send(x, make_float4(a, b, 0.0f, 0.0f), split, mine, round);
  const bool ok = exchange_wait(x, round);
  a = b = 0.0f;
#pragma unroll
  for (int r = 0; r < BN_MAX_CLUSTER; ++r)
    if (r < split) {
      const float4 v = x.slots[round & 1][r];
      a += v.x;
      b += v.y;
    }
  return ok;
}

// n values, their mean and the sum of their squared deviations from it
struct Moments { float n, mean, m2; };
// from the sums of the n values' x - shift and of its square
__device__ __forceinline__ Moments moments_of(float n, float inv_n, float shift, float s1, float s2) {
  const float d = s1 * inv_n, q = fmaf(-s1, d, s2);
  return {n, shift + d, q < 0.0f ? 0.0f : q};   // (NaN stays)
}
// how many values a warp, the CTA and the channel hold: the same for all channels
struct Counts { float n, inv_n, warp, inv_warp, inv_cta, cta, inv_all; };
__device__ __forceinline__ Counts channel_counts(Exchange& x, float n, float all) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = (int)blockDim.x >> 5;
  auto inv = [](float v) { return v > 0.0f ? 1.0f / v : 0.0f; };
  Counts c;
  c.n = n;
  c.warp = fb_warp_sum(n);
  if (lane == 0) x.warp_n[w] = c.warp;
  __syncthreads();
  c.cta = fb_warp_sum(lane < nw ? x.warp_n[lane] : 0.0f);
  c.inv_n = inv(n); c.inv_warp = inv(c.warp); c.inv_cta = inv(c.cta); c.inv_all = 1.0f / all;
  return c;
}
// The lanes' moments merged, valid in every lane.
__device__ __forceinline__ Moments warp_merge(const Moments& m, float n, float inv_n) {
  const float mean = fb_warp_sum(m.n * m.mean) * inv_n, d = m.mean - mean;
  return {n, mean, fb_warp_sum(fmaf(m.n * d, d, m.m2))};
}
// The channel's moments from those of all threads of the cluster, valid in every thread.
__device__ __forceinline__ bool channel_moments(Exchange& x, Moments& m, const Counts& c, int split, uint32_t mine, int round) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = (int)blockDim.x >> 5;
  m = warp_merge(m, c.warp, c.inv_warp);
  if (lane == 0) { x.sh[w] = m.mean; x.sh[32 + w] = m.m2; }
  __syncthreads();
  if (split == 1 || w == 0) {
    const bool there = lane < nw;
    m = warp_merge({there ? x.warp_n[lane] : 0.0f, there ? x.sh[lane] : 0.0f, there ? x.sh[32 + lane] : 0.0f}, c.cta, c.inv_cta);
  }
  if (split == 1) {
    __syncthreads();   // sh may be written again
    return true;
  }
  if (w == 0) exchange_send(x, make_float4(m.n, m.mean, m.m2, 0.0f), split, mine, round);
  const bool ok = exchange_wait(x, round);
  float4 v[BN_MAX_CLUSTER];
#pragma unroll
  for (int r = 0; r < BN_MAX_CLUSTER; ++r)
    if (r < split) v[r] = x.slots[round & 1][r];
  float s = 0.0f, q = 0.0f;
#pragma unroll
  for (int r = 0; r < BN_MAX_CLUSTER; ++r)
    if (r < split) s = fmaf(v[r].x, v[r].y, s);
  const float mean = s * c.inv_all;
#pragma unroll
  for (int r = 0; r < BN_MAX_CLUSTER; ++r)
    if (r < split) {
      const float d = v[r].y - mean;
      q += fmaf(v[r].x * d, d, v[r].z);
    }
  m.mean = mean;
  m.m2 = q;
  return ok;
}

// mean, 1 / std and running statistics of a channel of cnt values
struct ChannelStats { float mean, rs; };
__device__ __forceinline__ ChannelStats channel_stats(const Moments& m, float cnt, float eps, bool write, int64_t ch, float momentum,
                                                      float* save_mean, float* save_rstd, float* running_mean, float* running_var) {
  const float var = m.m2 / cnt;  // biased
  const float rs = rsqrtf(var + eps);
  if (write) {
    save_mean[ch] = m.mean;
    save_rstd[ch] = rs;
    if (running_mean != nullptr) {
      running_mean[ch] = (1.0f - momentum) * running_mean[ch] + momentum * m.mean;
      running_var[ch] = (1.0f - momentum) * running_var[ch] + momentum * var * (cnt / (cnt - 1.0f));
    }
  }
  return {m.mean, rs};
}

// ------------------------------------------------------------------------------ statistics ---
// One cluster of `split` CTAs per channel.
template <int W>
__global__ void __launch_bounds__(BN_THREADS)
bn_stats_kernel(const float* __restrict__ x, const Dims g, float eps, float momentum, float* __restrict__ save_mean,
                float* __restrict__ save_rstd, float* __restrict__ running_mean, float* __restrict__ running_var,
                int32_t* __restrict__ dev_err) {
  fb_after_previous();
  constexpr int U = 4;
  __shared__ Exchange ex;
  const int64_t ch = blockIdx.x / (unsigned)g.split;
  const int p = (int)(blockIdx.x % (unsigned)g.split);
  exchange_init(ex, g.split);
  constexpr int RUN = 256;   // values summed with one shift
  float shift = 0.0f, s1 = 0.0f, s2 = 0.0f;
  int k = 0;
  Moments own = {0.0f, 0.0f, 0.0f};
  auto fold = [&] {
    const Moments r = moments_of((float)k, 1.0f / (float)k, shift, s1, s2);
    fb_welford_merge(own.n, own.mean, own.m2, r.n, r.mean, r.m2);
    s1 = s2 = 0.0f;
    k = 0;
  };
  const Walk wk = make_walk<W>(g, p);
  each_piece<U>(wk, ch * g.s, [&](int, int64_t off, int m) {
    float v[U][W];
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (u < m) ld_piece<W>(x + off + u * wk.step, v[u]);
    if (k == 0) shift = v[0][0];
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (u < m)
#pragma unroll
        for (int e = 0; e < W; ++e) {
          const float a = v[u][e] - shift;
          s1 += a;
          s2 = fmaf(a, a, s2);
        }
    k += m * W;
    if (k >= RUN) fold();
  });
  if (k > 0) fold();
  const float cnt = (float)(g.s * g.n);
  const Counts counts = channel_counts(ex, own.n, cnt);
  const bool ok = channel_moments(ex, own, counts, g.split, (uint32_t)p, 0);
  channel_stats(own, cnt, eps, p == 0 && threadIdx.x == 0, ch, momentum, save_mean, save_rstd, running_mean, running_var);
  if (!ok && threadIdx.x == 0) atomicExch(dev_err, 2101);
  if (g.split > 1) cluster_sync_all();   // (no CTA leaves while another may still send to it)
}

// ------------------------------------------------------------- the whole training forward pass ---
// Cluster q of Q takes channels q, q + Q, ...; `depth` (1 .. 3) channels are held: each thread brings its own pieces with cp.async and
// reads nobody else's, so the copies need no barrier.
template <int W, int ACT>
__global__ void __launch_bounds__(BN_FWD_THREADS, 1)
bn_fwd_kernel(const float* __restrict__ x, const float* __restrict__ gamma, const float* __restrict__ beta, float* __restrict__ y,
              const Dims g, int depth, int slab, float eps, float momentum, float* __restrict__ save_mean, float* __restrict__ save_rstd,
              float* __restrict__ running_mean, float* __restrict__ running_var, int act, int32_t* __restrict__ dev_err) {
  fb_after_previous();
  extern __shared__ __align__(16) float cache[];   // [depth][piece][thread][W]
  __shared__ Exchange ex;
  const int p = (int)(blockIdx.x % (unsigned)g.split);
  const int64_t Q = gridDim.x / (unsigned)g.split, first = blockIdx.x / (unsigned)g.split;
  const float cnt = (float)(g.s * g.n);
  exchange_init(ex, g.split);
  const Walk wk = make_walk<W>(g, p);
  const int pieces = wk.mine * wk.cols, per = (int)blockDim.x * W;
  float* const own = cache + threadIdx.x * W;
  auto fetch = [&](int64_t ch, float* to) {
    if (ch < g.c) {
      uint32_t dst = smem_u32(to);
      each_piece<1>(wk, ch * g.s, [&](int, int64_t off, int) {
        if (W == 4) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(x + off) : "memory");
        else asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(x + off) : "memory");
        dst += (uint32_t)per * 4u;
      });
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  for (int d = 0; d < depth; ++d) fetch(first + d * Q, own + d * slab);
  const Counts counts = channel_counts(ex, (float)(pieces * W), cnt);
  // scale and bias: one channel ahead
  auto ahead = [&](const float* a, int64_t ch, float otherwise) { return a != nullptr && ch < g.c ? __ldg(a + ch) : otherwise; };
  float ga = ahead(gamma, first, 1.0f), be = ahead(beta, first, 0.0f);
  int d = 0, round = 0;
  bool ok = true;
  for (int64_t ch = first; ch < g.c; ch += Q, ++round) {
    const float ga1 = ahead(gamma, ch + Q, 1.0f), be1 = ahead(beta, ch + Q, 0.0f);
    if (depth == 3) asm volatile("cp.async.wait_group 2;" ::: "memory");
    else if (depth == 2) asm volatile("cp.async.wait_group 1;" ::: "memory");
    else asm volatile("cp.async.wait_group 0;" ::: "memory");
    float* const here = own + d * slab;
    float s1 = 0.0f, s2 = 0.0f;
    const float shift = pieces > 0 ? *here : 0.0f;
#pragma unroll 4
    for (int k = 0; k < pieces; ++k) {
      float v[W];
      ld_piece<W>(here + k * per, v);
#pragma unroll
      for (int e = 0; e < W; ++e) {
        const float a = v[e] - shift;
        s1 += a;
        s2 = fmaf(a, a, s2);
      }
    }
    Moments m = moments_of(counts.n, counts.inv_n, shift, s1, s2);
    ok = channel_moments(ex, m, counts, g.split, (uint32_t)p, round) && ok;
    const ChannelStats st = channel_stats(m, cnt, eps, p == 0 && threadIdx.x == 0, ch, momentum, save_mean, save_rstd, running_mean, running_var);
    const float sc = st.rs * ga;
    const float* src = here;
    each_piece<1>(wk, ch * g.s, [&](int, int64_t off, int) {
      float o[W];
      ld_piece<W>(src, o);
      src += per;
#pragma unroll
      for (int e = 0; e < W; ++e) o[e] = fb_act_apply_k<ACT>(act, fmaf(o[e] - st.mean, sc, be));
      st_piece<W>(y + off, o);
    });
    fetch(ch + depth * Q, here);
    d = d + 1 == depth ? 0 : d + 1;
    ga = ga1; be = be1;
  }
  if (!ok && threadIdx.x == 0) atomicExch(dev_err, 2101);
  if (g.split > 1) cluster_sync_all();   // (no CTA leaves while another may still send to it)
}

// ----------------------------------------------------------------------------- normalise pass ---
// rows of one chunk
__host__ __device__ __forceinline__ int bn_chunk(int nr) { return 8 * nr < BN_THREADS ? 8 * nr : BN_THREADS; }

// mean and rstd per channel; VAR: a variance is given instead of rstd
template <int W, bool VAR, int ACT>
__global__ void __launch_bounds__(BN_THREADS)
bn_apply_kernel(const float* __restrict__ x, const float* __restrict__ gamma, const float* __restrict__ beta,
                const float* __restrict__ mean, const float* __restrict__ rstd, float eps, float* __restrict__ y, int64_t s, int64_t c,
                int64_t rows, int tpr, int act) {
  fb_after_previous();
  constexpr int U = 4;
  __shared__ float3 par[BN_THREADS];   // mean, scale, shift of a chunk of rows: one thread each, not all threads for every row
  const int tx = threadIdx.x & (tpr - 1), ty = threadIdx.x / tpr, nr = BN_THREADS / tpr;
  const int chunk = bn_chunk(nr);
  for (int64_t r0 = (int64_t)blockIdx.x * chunk; r0 < rows; r0 += (int64_t)gridDim.x * chunk) {
    const int m = rows - r0 < chunk ? (int)(rows - r0) : chunk;
    __syncthreads();
    if ((int)threadIdx.x < m) {
      const int64_t r = r0 + threadIdx.x, ch = rows <= 0x7fffffff ? (int64_t)((uint32_t)r % (uint32_t)c) : r % c;
      const float q = __ldg(rstd + ch);
      par[threadIdx.x] = make_float3(__ldg(mean + ch), (VAR ? 1.0f / sqrtf(q + eps) : q) * (gamma ? __ldg(gamma + ch) : 1.0f), beta ? __ldg(beta + ch) : 0.0f);
    }
    __syncthreads();
    for (int k = ty; k < m; k += U * nr) {
      const float* xr = x + (r0 + k) * s;
      float* yr = y + (r0 + k) * s;
      for (int64_t j = (int64_t)tx * W; j < s; j += (int64_t)tpr * W) {
        float v[U][W];
#pragma unroll
        for (int u = 0; u < U; ++u)
          if (k + u * nr < m) ld_stream<W>(xr + u * nr * s + j, v[u]);
#pragma unroll
        for (int u = 0; u < U; ++u) {
          if (k + u * nr >= m) break;
          const float3 q = par[k + u * nr];
#pragma unroll
          for (int e = 0; e < W; ++e) v[u][e] = fb_act_apply_k<ACT>(act, fmaf(v[u][e] - q.x, q.y, q.z));
          st_stream<W>(yr + u * nr * s + j, v[u]);
        }
      }
    }
  }
}

// Short rows (less than 128 floats) whatever their alignment: the tensor as one run of float4 pieces, which may span rows.  s and
// c divide by multiplication (Granlund and Montgomery, "Division by invariant integers using multiplication").
struct FastDiv {
  uint32_t d, mul, sh1, sh2;
};
FastDiv fast_div(uint32_t d) {
  uint32_t l = 0;
  while (l < 32 && ((uint64_t)1 << l) < d) ++l;
  const uint64_t m = ((((uint64_t)1 << l) - d) << 32) / d + 1;
  return {d, (uint32_t)m, l < 1 ? l : 1, l < 1 ? 0 : l - 1};
}
__device__ __forceinline__ uint32_t quotient(const FastDiv& f, uint32_t n) {
  const uint32_t t = __umulhi(f.mul, n);
  return (t + ((n - t) >> f.sh1)) >> f.sh2;
}

template <bool VAR, int ACT>
__global__ void __launch_bounds__(BN_THREADS)
bn_apply_flat_kernel(const float* __restrict__ x, const float* __restrict__ gamma, const float* __restrict__ beta,
                     const float* __restrict__ mean, const float* __restrict__ rstd, float eps, float* __restrict__ y, const FastDiv fs,
                     const FastDiv fc, uint32_t total, int act) {
  fb_after_previous();
  constexpr int U = 2;
  for (uint32_t i = blockIdx.x * (U * BN_THREADS) + threadIdx.x; i < (total + 3) / 4; i += gridDim.x * (U * BN_THREADS)) {
    float v[U][4];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const uint32_t at = 4 * (i + u * BN_THREADS);
      if (at + 3 < total) {
        ld_piece<4>(x + at, v[u]);
      } else {
#pragma unroll
        for (int e = 0; e < 4; ++e) v[u][e] = at + e < total ? x[at + e] : 0.0f;
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const uint32_t at = 4 * (i + u * BN_THREADS);
      if (at >= total) break;
      const uint32_t row = quotient(fs, at);
      uint32_t pos = at - row * fs.d, ch = row - quotient(fc, row) * fc.d;
      float mu = 0.0f, sc = 0.0f, sf = 0.0f;
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        if (e == 0 || pos == 0) {
          const float q = __ldg(rstd + ch);
          mu = __ldg(mean + ch);
          sc = (VAR ? 1.0f / sqrtf(q + eps) : q) * (gamma ? __ldg(gamma + ch) : 1.0f);
          sf = beta ? __ldg(beta + ch) : 0.0f;
        }
        v[u][e] = fb_act_apply_k<ACT>(act, fmaf(v[u][e] - mu, sc, sf));
        if (++pos == fs.d) {
          pos = 0;
          if (++ch == fc.d) ch = 0;
        }
      }
      if (at + 3 < total) {
        st_piece<4>(y + at, v[u]);
      } else {
#pragma unroll
        for (int e = 0; e < 4; ++e)
          if (at + e < total) y[at + e] = v[u][e];
      }
    }
  }
}

// ----------------------------------------------------------------------------------- backward ---
// dgamma, dbeta and (coef != NULL) the means of dz and dz * xhat, with dz = dy_scale * dy * act'(gamma * xhat + beta); one cluster
// per channel
template <int W, int ACT, bool OWN>
__global__ void __launch_bounds__(BN_THREADS, 5)
bn_bwd_sums_kernel(const float* __restrict__ x, const float* __restrict__ dy, float dy_scale, const float* __restrict__ gamma,
                   const float* __restrict__ beta, const float* __restrict__ mean, const float* __restrict__ rstd, const Dims g,
                   float* __restrict__ coef, float* __restrict__ dgamma, float* __restrict__ dbeta, int act, int32_t* __restrict__ dev_err) {
  fb_after_previous();
  constexpr int U = OWN ? 4 : 2;
  __shared__ Exchange ex;
  exchange_init(ex, g.split);
  const int64_t ch = blockIdx.x / (unsigned)g.split;
  const int p = (int)(blockIdx.x % (unsigned)g.split);
  const float mu = __ldg(mean + ch), rs = __ldg(rstd + ch);
  const float ga = gamma ? __ldg(gamma + ch) : 1.0f, be = beta ? __ldg(beta + ch) : 0.0f;
  const float sc = rs * ga;   // (as the forward pass scales)
  float a1 = 0.0f, a2 = 0.0f;
  const Walk wk = make_walk<W>(g, p);
  each_piece<U>(wk, ch * g.s, [&](int, int64_t off, int m) {
    float v[U][W], d[U][W];
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (u < m) {
        ld_piece<W>(x + off + u * wk.step, v[u]);
        if (!OWN) ld_piece<W>(dy + off + u * wk.step, d[u]);
      }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (u >= m) break;
#pragma unroll
      for (int e = 0; e < W; ++e) {
        const float h = (v[u][e] - mu) * rs;
        float dz = (OWN ? fb_act_apply_k<ACT>(act, fmaf(v[u][e] - mu, sc, be)) : d[u][e]) * dy_scale;
        if (ACT != 0) dz = fb_act_bwd_k<ACT>(act, fmaf(h, ga, be), dz);
        a1 += dz;
        a2 = fmaf(dz, h, a2);
      }
    }
  });
  if (!channel_sums(ex, a1, a2, g.split, (uint32_t)p, 0) && threadIdx.x == 0) atomicExch(dev_err, 2101);
  if (p == 0 && threadIdx.x == 0) {
    if (dbeta) dbeta[ch] = a1;
    if (dgamma) dgamma[ch] = a2;
    if (coef) {
      const float cnt = (float)(g.s * g.n);
      coef[ch * 2 + 0] = a1 / cnt;
      coef[ch * 2 + 1] = a2 / cnt;
    }
  }
  if (g.split > 1) cluster_sync_all();   // (no CTA leaves while another may still send to it)
}

template <int W, int ACT>
__global__ void __launch_bounds__(BN_THREADS)
bn_bwd_apply_kernel(const float* __restrict__ x, const float* __restrict__ dy, const float* __restrict__ gamma,
                    const float* __restrict__ beta, const float* __restrict__ mean, const float* __restrict__ rstd,
                    const float* __restrict__ coef, float* __restrict__ dx, int64_t s, int64_t c, int64_t rows, int tpr, int act) {
  fb_after_previous();
  constexpr int U = 2;
  const int tx = threadIdx.x & (tpr - 1), ty = threadIdx.x / tpr, nr = BN_THREADS / tpr;
  for (int64_t r = (int64_t)blockIdx.x * nr + ty; r < rows; r += (int64_t)gridDim.x * nr) {
    const int64_t ch = rows <= 0x7fffffff ? (int64_t)((uint32_t)r % (uint32_t)c) : r % c;
    const float mu = __ldg(mean + ch), rs = __ldg(rstd + ch);
    const float ga = gamma ? __ldg(gamma + ch) : 1.0f, be = beta ? __ldg(beta + ch) : 0.0f;
    const float m1 = __ldg(coef + ch * 2), m2 = __ldg(coef + ch * 2 + 1), k = ga * rs;
    const int64_t base = r * s;
    for (int64_t j = (int64_t)tx * W; j < s; j += (int64_t)U * tpr * W) {
      float v[U][W], d[U][W];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int64_t ju = j + (int64_t)u * tpr * W;
        if (ju < s) {
          ld_stream<W>(x + base + ju, v[u]);
          ld_stream<W>(dy + base + ju, d[u]);
        }
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int64_t ju = j + (int64_t)u * tpr * W;
        if (ju >= s) break;
        float o[W];
#pragma unroll
        for (int e = 0; e < W; ++e) {
          const float h = (v[u][e] - mu) * rs;
          const float dz = ACT == 0 ? d[u][e] : fb_act_bwd_k<ACT>(act, fmaf(h, ga, be), d[u][e]);
          o[e] = k * (dz - m1 - h * m2);
        }
        st_stream<W>(dx + base + ju, o);
      }
    }
  }
}

// ------------------------------------------------------------------------------------ launches ---
int bn_tpr(int64_t pieces, int nt) {
  int t = 1;
  while (t < nt && t < pieces) t *= 2;
  return t;
}
// More CTAs per channel while the GPU has room for blocks and a block has four rows for each of its threads.
Dims bn_dims(const fb_ctx* ctx, int64_t s, int64_t c, int64_t n, int W, int nt, int64_t blocks) {
  Dims g = {s, c, n, 1, bn_tpr(s / W, nt)};
  while (g.split < BN_MAX_CLUSTER && c * g.split < blocks * ctx->sm_count && n >= 8 * (int64_t)g.split * (nt / g.tpr)) g.split *= 2;
  return g;
}

// A launch of so many clusters of g.split CTAs
template <typename K, typename... A>
int32_t bn_launch(K kern, cudaStream_t stream, const Dims& g, int64_t clusters, int nt, size_t smem, A... args) {
  FB_REQUIRE(clusters * g.split <= 0x7fffffff, FB_ERR_SHAPE, "batchnorm: too many channels");
  // (48 KB without asking, the kernels' static shared memory included)
  if (smem > 48 * 1024 - sizeof(Exchange)) FB_CUDA(fb_allow_smem(kern, BN_CACHE_MAX));
  cudaLaunchConfig_t lc;
  memset(&lc, 0, sizeof(lc));
  lc.gridDim = dim3((unsigned)(clusters * g.split), 1, 1);
  lc.blockDim = dim3((unsigned)nt, 1, 1);
  lc.dynamicSmemBytes = smem;
  lc.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[1] = fb_early_start();
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)g.split;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  lc.attrs = attr;
  lc.numAttrs = 2;
  FB_CUDA(cudaLaunchKernelEx(&lc, kern, args...));
  FB_LAUNCH_CHECK();
  return FB_OK;
}

unsigned bn_row_grid(const fb_ctx* ctx, int64_t rows, int tpr) {
  const int64_t nr = BN_THREADS / tpr;
  int64_t blocks = (rows + 2 * nr - 1) / (2 * nr);
  const int64_t cap = (int64_t)ctx->sm_count * 16;
  if (blocks > cap) blocks = cap;
  if (blocks < 1) blocks = 1;
  return (unsigned)blocks;
}

// f(W, activation kind) as compile-time constants
template <typename F>
auto bn_kind(bool vec, int act, F f) {
  return fb_act_kind(act, [&](auto k) {
    return vec ? f(std::integral_constant<int, 4>(), k) : f(std::integral_constant<int, 1>(), k);
  });
}

template <bool VAR>
int32_t bn_apply(fb_ctx* ctx, cudaStream_t stream, bool vec, const float* x, const float* gamma, const float* beta, const float* mean,
                 const float* rstd, float eps, float* y, int64_t s, int64_t c, int64_t n, int act) {
  if (s < 128 && s * c * n <= 0x7fffffff && fb_aligned16(x) && fb_aligned16(y)) {
    const int64_t pieces = (s * c * n + 3) / 4, per = 2 * BN_THREADS, blocks = (pieces + per - 1) / per, cap = (int64_t)ctx->sm_count * 16;
    fb_act_kind(act, [&](auto k) {
      fb_launch(bn_apply_flat_kernel<VAR, k.value>, (unsigned)(blocks < cap ? blocks : cap), BN_THREADS, 0, stream, x, gamma, beta, mean, rstd, eps, y, fast_div((uint32_t)s), fast_div((uint32_t)c), (uint32_t)(s * c * n), act);
    });
    FB_LAUNCH_CHECK();
    return FB_OK;
  }
  const int tpr = bn_tpr(vec ? s / 4 : s, BN_THREADS);
  bn_kind(vec, act, [&](auto W, auto k) {
    const int64_t chunk = bn_chunk(BN_THREADS / tpr), blocks = (c * n + chunk - 1) / chunk, cap = (int64_t)ctx->sm_count * 32;
    fb_launch(bn_apply_kernel<W.value, VAR, k.value>, (unsigned)(blocks < cap ? blocks : cap), BN_THREADS, 0, stream, x, gamma, beta, mean, rstd, eps, y, s, c, c * n, tpr, act);
  });
  FB_LAUNCH_CHECK();
  return FB_OK;
}

// y = act(BatchNorm(x)) with batch statistics, which are saved; running statistics are updated where given
int32_t bn_fwd_batch(fb_ctx* ctx, cudaStream_t stream, const float* x, const float* gamma, const float* beta, float* running_mean,
                     float* running_var, float* y, float* save_mean, float* save_rstd, int64_t s, int64_t c, int64_t n, float eps,
                     float momentum, int act) {
  const bool vec = (s % 4 == 0) && fb_aligned16(x) && fb_aligned16(y);
  const int W = vec ? 4 : 1;
  // few values per channel: smaller blocks
  const int nt = s * n > 2048 * W ? BN_FWD_THREADS : BN_THREADS;
  Dims g = {s, c, n, 1, bn_tpr(s / W, nt)};
  auto bytes = [&] {
    const int64_t rows = (int64_t)g.split * (nt / g.tpr);
    return (size_t)((n + rows - 1) / rows * ((s / W + g.tpr - 1) / g.tpr)) * nt * W * sizeof(float);
  };
  int lg = 0;
  // two channels at least in a CTA's shared memory, and every SM with a CTA, as long as there are rows for more CTAs: large images in
  // small batches would wait for clusters of which most CTAs own nothing (160 x 160 x 64 channels: one sample 29 us with eight CTAs, now
  // 7.6; two 29 and 10.8; four 30 and 18; 224 x 224: one 45 and 11, four 47 and 28)
  while (g.split < BN_MAX_CLUSTER && n > (int64_t)g.split * (nt / g.tpr) && (2 * bytes() > BN_CACHE_MAX || (c * g.split < ctx->sm_count && n >= 8 * (int64_t)g.split * (nt / g.tpr)))) {
    g.split *= 2;
    ++lg;
  }
  const size_t slab = bytes();
  if (slab <= BN_CACHE_MAX) {
    const int64_t resident = ctx->clusters[lg] > 0 ? ctx->clusters[lg] : 1, clusters = c < resident ? c : resident;
    const int64_t rounds = (c + clusters - 1) / clusters;
    int depth = (int)(BN_CACHE_MAX / slab);
    depth = depth > 3 ? 3 : depth;
    depth = depth > rounds ? (int)rounds : depth;
    return bn_kind(vec, act, [&](auto w, auto k) {
      return bn_launch(bn_fwd_kernel<w.value, k.value>, stream, g, clusters, nt, slab * depth, x, gamma, beta, y, g, depth, (int)(slab / sizeof(float)), eps,
                       momentum, save_mean, save_rstd, running_mean, running_var, act, ctx->dev_error);
    });
  }
  g = bn_dims(ctx, s, c, n, W, BN_THREADS, 12);
  const int32_t st = bn_kind(vec, FB_ACT_IDENTITY, [&](auto w, auto) {
    return bn_launch(bn_stats_kernel<w.value>, stream, g, c, BN_THREADS, 0, x, g, eps, momentum, save_mean, save_rstd, running_mean, running_var,
                     ctx->dev_error);
  });
  return st != FB_OK ? st : bn_apply<false>(ctx, stream, vec, x, gamma, beta, save_mean, save_rstd, eps, y, s, c, n, act);
}

// dy == NULL: the cotangent is dy_scale times the layer's output, which the kernel makes from x instead of reading it
int32_t bn_bwd_sums(fb_ctx* ctx, cudaStream_t stream, bool vec, const float* x, const float* dy, float dy_scale, const float* gamma,
                    const float* beta, const float* mean, const float* rstd, float* coef, float* dgamma, float* dbeta, int64_t s,
                    int64_t c, int64_t n, int act) {
  const Dims g = bn_dims(ctx, s, c, n, vec ? 4 : 1, BN_THREADS, 12);
  return bn_kind(vec, act, [&](auto w, auto k) {
    return bn_launch(dy != nullptr ? bn_bwd_sums_kernel<w.value, k.value, false> : bn_bwd_sums_kernel<w.value, k.value, true>, stream, g, c, BN_THREADS, 0, x, dy,
                     dy_scale, gamma, beta, mean, rstd, g, coef, dgamma, dbeta, act, ctx->dev_error);
  });
}

int32_t bn_check(const char* fn, int64_t s, int64_t c, int64_t n, int act) {
  FB_REQUIRE(s >= 1 && c >= 1 && n >= 0, FB_ERR_SHAPE, "%s: bad shape s=%lld c=%lld n=%lld", fn, (long long)s,
             (long long)c, (long long)n);
  FB_REQUIRE(c <= 0x7fffffff, FB_ERR_SHAPE, "%s: too many channels", fn);
  FB_REQUIRE(fb_act_valid(act), FB_ERR_INVALID_ARG, "%s: unknown activation %d", fn, act);
  return FB_OK;
}

}  // namespace

FB_API int32_t fb_batchnorm_fwd_train(fb_ctx* ctx, void* stream_, const float* x, const float* gamma,
                                      const float* beta, float* running_mean, float* running_var, float* y,
                                      float* save_mean, float* save_rstd, int64_t s, int64_t c, int64_t n,
                                      float eps, float momentum, int32_t act, int32_t track_stats) {
  FB_CHECK_CTX(ctx);
  cudaStream_t stream = (cudaStream_t)stream_;
  int32_t st = bn_check("fb_batchnorm_fwd_train", s, c, n, act);
  if (st != FB_OK) return st;
  FB_REQUIRE((gamma == nullptr) == (beta == nullptr), FB_ERR_INVALID_ARG, "fb_batchnorm_fwd_train: gamma and beta must both be given or both NULL");
  FB_REQUIRE(s * n > 1, FB_ERR_SHAPE,
             "fb_batchnorm_fwd_train: BatchNorm expected more than 1 value per channel when training, got s*n = %lld",
             (long long)(s * n));
  FB_REQUIRE(x && y && save_mean && save_rstd, FB_ERR_INVALID_ARG, "fb_batchnorm_fwd_train: NULL pointer");
  FB_REQUIRE((running_mean == nullptr) == (running_var == nullptr), FB_ERR_INVALID_ARG, "fb_batchnorm_fwd_train: running_mean and running_var must both be given or both NULL");
  const bool upd = track_stats != 0 && running_mean != nullptr;
  return bn_fwd_batch(ctx, stream, x, gamma, beta, upd ? running_mean : nullptr, upd ? running_var : nullptr, y, save_mean, save_rstd, s,
                      c, n, eps, momentum, act);
}

FB_API int32_t fb_batchnorm_fwd_infer(fb_ctx* ctx, void* stream_, const float* x, const float* gamma,
                                      const float* beta, const float* running_mean, const float* running_var,
                                      float* y, int64_t s, int64_t c, int64_t n, float eps, int32_t act) {
  FB_CHECK_CTX(ctx);
  cudaStream_t stream = (cudaStream_t)stream_;
  int32_t st = bn_check("fb_batchnorm_fwd_infer", s, c, n, act);
  if (st != FB_OK) return st;
  FB_REQUIRE((gamma == nullptr) == (beta == nullptr), FB_ERR_INVALID_ARG, "fb_batchnorm_fwd_infer: gamma and beta must both be given or both NULL");
  if (n == 0) return FB_OK;
  FB_REQUIRE(x && y, FB_ERR_INVALID_ARG, "fb_batchnorm_fwd_infer: NULL pointer");
  if (running_mean != nullptr && running_var != nullptr) {
    const bool vec = (s % 4 == 0) && fb_aligned16(x) && fb_aligned16(y);
    return bn_apply<true>(ctx, stream, vec, x, gamma, beta, running_mean, running_var, eps, y, s, c, n, act);
  }
  float* ws = (float*)fb_scratch(ctx, stream, (size_t)c * 2 * sizeof(float));
  if (!ws) return FB_ERR_ALLOC;
  return bn_fwd_batch(ctx, stream, x, gamma, beta, nullptr, nullptr, y, ws, ws + c, s, c, n, eps, 0.0f, act);
}

FB_API int32_t fb_batchnorm_bwd(fb_ctx* ctx, void* stream_, const float* x, const float* gamma,
                                const float* beta, const float* save_mean, const float* save_rstd,
                                const float* dy, float* dx, float* dgamma, float* dbeta, int64_t s, int64_t c,
                                int64_t n, int32_t act) {
  FB_CHECK_CTX(ctx);
  cudaStream_t stream = (cudaStream_t)stream_;
  int32_t st = bn_check("fb_batchnorm_bwd", s, c, n, act);
  if (st != FB_OK) return st;
  FB_REQUIRE((gamma == nullptr) == (beta == nullptr), FB_ERR_INVALID_ARG, "fb_batchnorm_bwd: gamma and beta must both be given or both NULL");
  FB_REQUIRE(n >= 1, FB_ERR_SHAPE, "fb_batchnorm_bwd: empty batch");
  FB_REQUIRE(x && save_mean && save_rstd && dy && dx, FB_ERR_INVALID_ARG, "fb_batchnorm_bwd: NULL pointer");
  float* coef = (float*)fb_scratch(ctx, stream, (size_t)c * 2 * sizeof(float));
  if (!coef) return FB_ERR_ALLOC;
  const bool vec = (s % 4 == 0) && fb_aligned16(x) && fb_aligned16(dy) && fb_aligned16(dx);
  st = bn_bwd_sums(ctx, stream, vec, x, dy, 1.0f, gamma, beta, save_mean, save_rstd, coef, dgamma, dbeta, s, c, n, act);
  if (st != FB_OK) return st;
  const int tpr = bn_tpr(vec ? s / 4 : s, BN_THREADS);
  bn_kind(vec, act, [&](auto w, auto k) {
    fb_launch(bn_bwd_apply_kernel<w.value, k.value>, bn_row_grid(ctx, c * n, tpr), BN_THREADS, 0, stream, x, dy, gamma, beta, save_mean, save_rstd, coef, dx, s, c, c * n, tpr, act);
  });
  FB_LAUNCH_CHECK();
  return FB_OK;
}

FB_API int32_t fb_batchnorm_bwd_params(fb_ctx* ctx, void* stream_, const float* x, const float* gamma, const float* beta,
                                       const float* save_mean, const float* save_rstd, const float* dy, float dy_scale,
                                       float* dgamma, float* dbeta, int64_t s, int64_t c, int64_t n, int32_t act) {
  FB_CHECK_CTX(ctx);
  int32_t st = bn_check("fb_batchnorm_bwd_params", s, c, n, act);
  if (st != FB_OK) return st;
  FB_REQUIRE((gamma == nullptr) == (beta == nullptr), FB_ERR_INVALID_ARG, "fb_batchnorm_bwd_params: gamma and beta must both be given or both NULL");
  FB_REQUIRE(n >= 1, FB_ERR_SHAPE, "fb_batchnorm_bwd_params: empty batch");
  FB_REQUIRE(x && save_mean && save_rstd && dy && dgamma && dbeta, FB_ERR_INVALID_ARG, "fb_batchnorm_bwd_params: NULL pointer");
  const bool vec = (s % 4 == 0) && fb_aligned16(x) && fb_aligned16(dy);
  return bn_bwd_sums(ctx, (cudaStream_t)stream_, vec, x, dy, dy_scale, gamma, beta, save_mean, save_rstd, nullptr, dgamma, dbeta, s, c, n, act);
}

FB_API int32_t fb_batchnorm_bwd_params_own(fb_ctx* ctx, void* stream_, const float* x, const float* gamma, const float* beta,
                                           const float* save_mean, const float* save_rstd, float y_scale, float* dgamma, float* dbeta,
                                           int64_t s, int64_t c, int64_t n, int32_t act) {
  FB_CHECK_CTX(ctx);
  int32_t st = bn_check("fb_batchnorm_bwd_params_own", s, c, n, act);
  if (st != FB_OK) return st;
  FB_REQUIRE((gamma == nullptr) == (beta == nullptr), FB_ERR_INVALID_ARG, "fb_batchnorm_bwd_params_own: gamma and beta must both be given or both NULL");
  FB_REQUIRE(n >= 1, FB_ERR_SHAPE, "fb_batchnorm_bwd_params_own: empty batch");
  FB_REQUIRE(x && save_mean && save_rstd && dgamma && dbeta, FB_ERR_INVALID_ARG, "fb_batchnorm_bwd_params_own: NULL pointer");
  const bool vec = (s % 4 == 0) && fb_aligned16(x);
  return bn_bwd_sums(ctx, (cudaStream_t)stream_, vec, x, nullptr, y_scale, gamma, beta, save_mean, save_rstd, nullptr, dgamma, dbeta, s, c, n, act);
}
