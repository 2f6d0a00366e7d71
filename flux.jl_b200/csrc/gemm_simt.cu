// fp32 FMA GEMM for the products the tensor-core kernel does not take or is too coarse for: few or skinny tiles (one
// sample through a layer, the 10-class output layer, the input projection of a short sequence) and operands whose
// rows are not 16-byte aligned.
//
// What bounds it: such a product is a few microseconds of loads and FMAs if the whole chip takes part, and its latency
// if it does not.  A grid of plain output tiles leaves most SMs idle (a 784 => 512 layer at batch 1 has 8 tiles of
// 64 columns; the 10-class layer at batch 1024 one column tile with K = 512 walked serially), so K is cut over a
// cluster of up to 8 CTAs: every CTA accumulates its K range, leaves its tile in shared memory, and after a cluster
// barrier the CTAs add up one slice of the tile each out of their peers' shared memory, in rank order (no workspace,
// no atomics: the result does not depend on timing).  Inside a CTA narrow tiles (16 rows or columns) are computed by
// four thread groups that share the k values of a stage.  Operand tiles travel by cp.async (16 bytes where rows are
// aligned, else 4) through three stages and stay in their global layout ([k][m] or [m][k]); both are read by
// 128-bit shared loads, 8 of them per 64 FMAs.
#include "common.cuh"

namespace {

constexpr int THREADS = 256, BK = 32, STAGES = 3;

__device__ __forceinline__ uint32_t s_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
// copies `bytes` (<= SIZE) and zero-fills the rest; nothing is read when bytes == 0
__device__ __forceinline__ void cp16(uint32_t dst, const float* src, int bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp4(uint32_t dst, const float* src, int bytes) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}

// Brings the BX x BK tile at (x0, k) of an operand with X rows (m or n) into shared memory, k advancing by BK from call
// to call.  MN: global [k][x], shared [BK][BX + 4]; otherwise global [x][k], shared [BX][BK + 4].  A thread's pieces lie
// RPI rows apart in one column, so that a call costs an add and a compare for each of them.
template <int BX, bool MN, bool VEC>
struct TileLoader {
  static constexpr int W = MN ? BX : BK, R = MN ? BK : BX;   // contiguous extent, rows
  static constexpr int E = VEC ? 4 : 1, CW = W / E, RPI = THREADS / CW, NI = (R + RPI - 1) / RPI;
  const float* p;      // piece 0 of the next tile
  int64_t step;        // floats between pieces
  int64_t k;           // first k of this thread's pieces: of the column (K-major) or of piece 0 (MN)
  uint32_t rows;       // K-major: bit i = row of piece i exists
  int bytes;           // MN: bytes of the column that exist
  int off;             // shared-memory offset of piece 0, floats (negative: this thread has no piece)
  __device__ __forceinline__ void init(const float* g, int64_t ld, int64_t x0, int64_t X, int64_t k0) {
    const int r = threadIdx.x / CW, c = (threadIdx.x % CW) * E;
    off = r < R ? r * (W + 4) + c : -1;
    step = (int64_t)RPI * ld;
    if (MN) {
      p = g + (k0 + r) * ld + x0 + c;
      k = k0 + r;
      const int64_t left = X - (x0 + c);
      bytes = left <= 0 ? 0 : left >= E ? 4 * E : (int)left * 4;
    } else {
      p = g + (x0 + r) * ld + k0 + c;
      k = k0 + c;
      rows = 0;
#pragma unroll
      for (int i = 0; i < NI; ++i)
        if (x0 + r + i * RPI < X) rows |= 1u << i;
    }
  }
  __device__ __forceinline__ void load(float* s, const float* g, int64_t ld, int64_t kend) {
    if (off >= 0) {
      const uint32_t dst = s_addr(s + off);
      int kb = 0;
      if (!MN) {
        const int64_t left = kend - k;
        kb = left <= 0 ? 0 : left >= E ? 4 * E : (int)left * 4;
      }
#pragma unroll
      for (int i = 0; i < NI; ++i) {
        const int b = MN ? (k + i * RPI < kend ? bytes : 0) : ((rows >> i) & 1u ? kb : 0);
        const float* src = b > 0 ? p + i * step : g;
        if (VEC) cp16(dst + (uint32_t)(i * RPI * (W + 4) * 4), src, b);
        else cp4(dst + (uint32_t)(i * RPI * (W + 4) * 4), src, b);
      }
    }
    p += MN ? (int64_t)BK * ld : (int64_t)BK;
    k += BK;
  }
};

// BM x BN tile; a thread owns TM x TN outputs and KG = 256 / (BM * BN / (TM * TN)) thread groups share the k values of a
// stage.  Row i of thread row tr is tr + i * BM / TM for a K-major operand (whose shared rows are BK + 4 floats apart, so
// that neighbouring thread rows fall on different banks) and i / 4 * 4 * BM / TM + 4 * tr + i % 4 for an MN-major one;
// columns alike.
template <int BM, int BN, int TM, int TN, bool A_MN, bool B_MN, bool AV, bool BV>
__global__ void __launch_bounds__(THREADS)
gemm_fma_kernel(const float* __restrict__ A, int64_t lda, const float* __restrict__ B, int64_t ldb, float* __restrict__ C, int64_t ldc,
                float* __restrict__ Z, const float* __restrict__ bias_n, const float* __restrict__ bias_m, int64_t M, int64_t N,
                int64_t K, int act, int accumulate, int splits, int64_t kper, int64_t tiles_n) {
  fb_after_previous();
  fb_let_next_start();
  constexpr int TR = BM / TM, TC = BN / TN, KG = THREADS / (TR * TC), KPG = BK / KG;
  static_assert(KG >= 1 && KPG >= 4, "a group needs four k values per stage");
  constexpr int AS = A_MN ? BK * (BM + 4) : BM * (BK + 4), BS = B_MN ? BK * (BN + 4) : BN * (BK + 4);
  extern __shared__ __align__(16) float sm[];
  const int split = (int)(blockIdx.x % (unsigned)splits);
  const int64_t tile = blockIdx.x / (unsigned)splits;
  const int64_t m0 = tile / tiles_n * BM, n0 = tile % tiles_n * BN;
  const int64_t kbeg = (int64_t)split * kper, kend = kbeg + kper < K ? kbeg + kper : K;
  const int nst = kend > kbeg ? (int)((kend - kbeg + BK - 1) / BK) : 0;
  const int kg = threadIdx.x / (TR * TC), tt = threadIdx.x % (TR * TC);
  // a warp covers 4 thread rows x 8 thread columns where the tile allows
  constexpr int WC = TC < 8 ? TC : 8, WR = 32 / WC;
  const int wv = tt / 32, ln = tt % 32;
  const int tr = (wv / (TC / WC)) * WR + ln / WC, tc = (wv % (TC / WC)) * WC + ln % WC;

  TileLoader<BM, A_MN, AV> la;
  TileLoader<BN, B_MN, BV> lb;
  la.init(A, lda, m0, M, kbeg);
  lb.init(B, ldb, n0, N, kbeg);
  auto load = [&](int st) {
    float* sa = sm + (st % STAGES) * (AS + BS);
    la.load(sa, A, lda, kend);
    lb.load(sa + AS, B, ldb, kend);
  };
  float acc[TM][TN];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = 0.0f;
#pragma unroll
  for (int st = 0; st < STAGES - 1; ++st) {
    if (st < nst) load(st);
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  for (int st = 0; st < nst; ++st) {
    asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
    __syncthreads();
    if (st + STAGES - 1 < nst) load(st + STAGES - 1);
    asm volatile("cp.async.commit_group;" ::: "memory");
    const float* sa = sm + (st % STAGES) * (AS + BS);
    const float* sb = sa + AS;
#pragma unroll
    for (int k4 = 0; k4 < KPG; k4 += 4) {
      const int k = kg * KPG + k4;
      float4 a[TM], b[TN];   // MN-major: [k][row quad]; K-major: [row], four k values each
#pragma unroll
      for (int i = 0; i < TM; ++i)
        a[i] = A_MN ? *(const float4*)(sa + (k + i / (TM / 4)) * (BM + 4) + (i % (TM / 4)) * 4 * TR + 4 * tr)
                    : *(const float4*)(sa + (tr + i * TR) * (BK + 4) + k);
#pragma unroll
      for (int j = 0; j < TN; ++j)
        b[j] = B_MN ? *(const float4*)(sb + (k + j / (TN / 4)) * (BN + 4) + (j % (TN / 4)) * 4 * TC + 4 * tc)
                    : *(const float4*)(sb + (tc + j * TC) * (BK + 4) + k);
      const float* af = (const float*)a;
      const float* bf = (const float*)b;
#pragma unroll
      for (int kk = 0; kk < 4; ++kk)
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
          for (int j = 0; j < TN; ++j)
            acc[i][j] = fmaf(A_MN ? af[TM * kk + i] : af[4 * i + kk], B_MN ? bf[TN * kk + j] : bf[4 * j + kk], acc[i][j]);
    }
  }
  auto row_of = [&](int i) { return A_MN ? i / 4 * 4 * TR + 4 * tr + i % 4 : tr + i * TR; };
  auto col_of = [&](int j) { return B_MN ? j / 4 * 4 * TC + 4 * tc + j % 4 : tc + j * TC; };
  auto emit = [&](int64_t gm, int64_t gn, float v) {
    if (accumulate) v += C[gm * ldc + gn];
    if (bias_n) v += __ldg(bias_n + gn);
    if (bias_m) v += __ldg(bias_m + gm);
    if (Z) Z[gm * ldc + gn] = v;
    C[gm * ldc + gn] = fb_act_apply(act, v);
  };
  // the groups' partial tiles [KG][BM][BN + 4] in shared memory, added up into the first ...
  constexpr int LD = BN + 4;
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      float* d = sm + (kg * BM + row_of(i)) * LD + col_of(j);
      if (B_MN && j % 4 == 0) *(float4*)d = make_float4(acc[i][j], acc[i][j + 1 < TN ? j + 1 : j], acc[i][j + 2 < TN ? j + 2 : j], acc[i][j + 3 < TN ? j + 3 : j]);
      else if (!B_MN) *d = acc[i][j];
    }
  __syncthreads();
  constexpr int QUADS = BM * BN / 4;
  auto quad = [&](int e) { return (e / (BN / 4)) * LD + (e % (BN / 4)) * 4; };
  auto finish = [&](int e, float4 x) {
    const int64_t gm = m0 + e / (BN / 4), gn = n0 + (e % (BN / 4)) * 4;
    const float v[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (gm < M && gn + i < N) emit(gm, gn + i, v[i]);
  };
#pragma unroll
  for (int e = threadIdx.x; e < QUADS; e += THREADS) {
    const int o = quad(e);
    float4 x[KG];
#pragma unroll
    for (int g = 0; g < KG; ++g) x[g] = *(const float4*)(sm + g * BM * LD + o);
#pragma unroll
    for (int g = 1; g < KG; ++g) { x[0].x += x[g].x; x[0].y += x[g].y; x[0].z += x[g].z; x[0].w += x[g].w; }
    if (splits == 1) finish(e, x[0]);
    else *(float4*)(sm + o) = x[0];
  }
  if (splits == 1) return;
  // ... then every CTA of the cluster finishes one slice of the tile out of all peers' sums, in rank order
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
  const int per = QUADS / splits;   // splits is a power of two <= 8
  for (int q = threadIdx.x; q < per; q += THREADS) {
    const int e = split * per + q;
    float4 x[8];   // all peers' loads in flight at once
#pragma unroll
    for (int s = 0; s < 8; ++s)
      if (s < splits) {
        uint32_t a;
        asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(s_addr(sm + quad(e))), "r"(s));
        asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(x[s].x), "=f"(x[s].y), "=f"(x[s].z), "=f"(x[s].w) : "r"(a) : "memory");
      }
#pragma unroll
    for (int s = 1; s < 8; ++s)
      if (s < splits) { x[0].x += x[s].x; x[0].y += x[s].y; x[0].z += x[s].z; x[0].w += x[s].w; }
    finish(e, x[0]);
  }
  // a peer may still be reading this CTA's tile
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

template <int BM, int BN, int TM, int TN, bool A_MN, bool B_MN, bool AV, bool BV>
int32_t launch_fma_variant(fb_ctx* ctx, cudaStream_t stream, const fb_gemm_args& a, int splits) {
  constexpr size_t STAGE = (size_t)((A_MN ? BK * (BM + 4) : BM * (BK + 4)) + (B_MN ? BK * (BN + 4) : BN * (BK + 4))) * 4;
  constexpr size_t PART = (size_t)THREADS * TM * TN / BN * (BN + 4) * 4;
  constexpr size_t SMEM = STAGES * STAGE > PART ? STAGES * STAGE : PART;
  const int64_t tiles_n = (a.N + BN - 1) / BN, tiles = tiles_n * ((a.M + BM - 1) / BM);
  const int64_t kper = ((a.K + BK - 1) / BK + splits - 1) / splits * BK;   // whole stages
  FB_REQUIRE(tiles * splits <= 0x7fffffff, FB_ERR_SHAPE, "gemm: too many tiles for the FMA kernel (M=%lld N=%lld)", (long long)a.M,
             (long long)a.N);
  auto kern = gemm_fma_kernel<BM, BN, TM, TN, A_MN, B_MN, AV, BV>;
  static thread_local int prepared = -1;
  if (prepared != ctx->device) {
    FB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 120 * 1024));
    FB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared));
    prepared = ctx->device;
  }
  cudaLaunchConfig_t lc;
  memset(&lc, 0, sizeof(lc));
  lc.gridDim = dim3((unsigned)(tiles * splits), 1, 1);
  lc.blockDim = dim3(THREADS, 1, 1);
  // The CTAs of a cluster are packed on as few SMs as hold them while others idle; asking for half an SM's shared memory
  // gives every CTA an SM of its own.
  lc.dynamicSmemBytes = splits > 1 ? 118 * 1024 : SMEM;
  lc.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[1] = fb_early_start();
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)splits;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  lc.attrs = splits > 1 ? attr : attr + 1;
  lc.numAttrs = splits > 1 ? 2 : 1;
  FB_CUDA(cudaLaunchKernelEx(&lc, kern, a.A, a.lda, a.B, a.ldb, a.C, a.ldc, a.Z, a.bias_n, a.bias_m, a.M, a.N, a.K, a.act, a.accumulate,
                             splits, kper, tiles_n));
  FB_LAUNCH_CHECK();
  return FB_OK;
}

template <int BM, int BN, int TM, int TN, bool A_MN, bool B_MN>
int32_t launch_fma(fb_ctx* ctx, cudaStream_t stream, const fb_gemm_args& a, int splits) {
  const bool av = a.lda % 4 == 0 && fb_aligned16(a.A), bv = a.ldb % 4 == 0 && fb_aligned16(a.B);
  if (av) return bv ? launch_fma_variant<BM, BN, TM, TN, A_MN, B_MN, true, true>(ctx, stream, a, splits) : launch_fma_variant<BM, BN, TM, TN, A_MN, B_MN, true, false>(ctx, stream, a, splits);
  return bv ? launch_fma_variant<BM, BN, TM, TN, A_MN, B_MN, false, true>(ctx, stream, a, splits) : launch_fma_variant<BM, BN, TM, TN, A_MN, B_MN, false, false>(ctx, stream, a, splits);
}

template <int BM, int BN, int TM, int TN>
int32_t launch_fma_layout(fb_ctx* ctx, cudaStream_t stream, const fb_gemm_args& a, int splits) {
  if (a.a_mn_major) return a.b_mn_major ? launch_fma<BM, BN, TM, TN, true, true>(ctx, stream, a, splits) : launch_fma<BM, BN, TM, TN, true, false>(ctx, stream, a, splits);
  return a.b_mn_major ? launch_fma<BM, BN, TM, TN, false, true>(ctx, stream, a, splits) : launch_fma<BM, BN, TM, TN, false, false>(ctx, stream, a, splits);
}

}  // namespace

// Tile and K split by the smallest modelled time: waves of CTAs (clusters) x stages of 32 k-values x the cost of a stage,
// measured on B200 at 1.0 us for a 64 x 64 tile, 0.55 for 32 x 64 and 0.3 for the 16-wide ones (taken where a dimension
// is at most 16 and a wider tile would compute padding), plus 1 us for a cluster's reduction.  About 15 / 33 / 74 clusters
// of 8 / 4 / 2 CTAs with an SM each are resident at once.
namespace {
struct FmaPlan {
  int thin, half, splits;   // 16-wide tile of rows (1) or columns (2); 32 x 64 instead of 64 x 64; CTAs that share K
  double time;
};
FmaPlan plan_fma(const fb_ctx* ctx, const fb_gemm_args& a) {
  const int thin = a.M <= 16 ? 1 : a.N <= 16 ? 2 : 0;
  const int64_t stages = (a.K + BK - 1) / BK;
  const int slots[4] = {ctx->sm_count, ctx->sm_count / 2, ctx->sm_count * 33 / 148, ctx->sm_count * 15 / 148};
  int best_half = 0, best_splits = 1;
  double best_t = 1e30;
  for (int half = 0; half < (thin ? 1 : 2); ++half) {
    const int64_t bm = thin == 1 ? 16 : thin == 2 ? 64 : half ? 32 : 64, bn = thin == 2 ? 16 : 64;
    const double cost = thin ? 0.3 : half ? 0.55 : 1.0;
    const int64_t tiles = ((a.M + bm - 1) / bm) * ((a.N + bn - 1) / bn);
    for (int lg = 0; lg < 4; ++lg) {
      const int s = 1 << lg;
      if (s > 1 && stages < s) break;
      double waves = (double)((tiles + slots[lg] - 1) / slots[lg]);
      if (s == 1 && waves > 1.0) waves = (double)tiles / slots[0];   // two CTAs share an SM
      const double t = waves * (double)((stages + s - 1) / s) * cost + (s > 1 ? 1.0 : 0.0);
      if (t < best_t) { best_t = t; best_half = half; best_splits = s; }
    }
  }
  return {thin, best_half, best_splits, best_t};
}
}  // namespace

double fb_gemm_simt_time(const fb_ctx* ctx, const fb_gemm_args& a) { return plan_fma(ctx, a).time; }

int32_t fb_gemm_simt_launch(fb_ctx* ctx, cudaStream_t stream, const fb_gemm_args& a) {
  if (a.M == 0 || a.N == 0) return FB_OK;
  const FmaPlan p = plan_fma(ctx, a);
  if (p.thin == 1) return launch_fma_layout<16, 64, 4, 4>(ctx, stream, a, p.splits);
  if (p.thin == 2) return launch_fma_layout<64, 16, 4, 4>(ctx, stream, a, p.splits);
  if (p.half) return launch_fma_layout<32, 64, 4, 4>(ctx, stream, a, p.splits);
  return launch_fma_layout<64, 64, 4, 4>(ctx, stream, a, p.splits);
}
