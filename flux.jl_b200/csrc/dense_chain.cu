// Consecutive Dense layers for a few columns, in one launch: a request to a served model.
//
// Layer by layer such a call is a string of launches of 4 - 5 us, each with its own start, its own wait for weights from L2 and a
// host call of 7 us before it.  Here a cluster of 16 CTAs keeps up to 4 columns to itself: CTA r owns one slice of every layer's
// outputs, results go to all 16 shared memories (distributed shared memory) and one cluster barrier separates two layers.  The weights of
// a slice stream through a ring of stages (cp.async); the ring does not stop at a layer's end, so that the next layer's weights are there
// when its inputs are.  Further columns are further clusters.
//
// What bounds it: the start (about 4 us), 1/16 of the weights through one SM (1 MB a layer: 2 us) and about 1 us a layer for the sum over
// the warps, the pushes and the barrier.  One column, us of device time and of a call that follows others: 784 -> 512 -> 512 -> 10
// (2.7 MB) 14.3 and 24 layer by layer, 11.1 and 12.4 here; with two more layers of 512 23.2 and 45, 17.8 and 20; 64 -> 64 -> 64 -> 7
// 9.3 and 28, 6.9 and 10.
#include "common.cuh"

namespace {

constexpr int DC_CTAS = 16, DC_THREADS = 512, DC_WARPS = DC_THREADS / 32, DC_MAX_LAYERS = 8;
constexpr int DC_STAGES = 5, DC_STAGE = 24 * 1024;      // bytes
constexpr int DC_WIDTH = 8192;                          // floats of one layer's inputs: width x columns
constexpr int DC_MAX_SLICE = 128;                       // outputs of a CTA
static_assert(DC_CTAS == DC_WARPS && DC_WIDTH / DC_CTAS <= DC_THREADS, "a warp per destination, a thread per output");
constexpr int DC_SMEM = DC_STAGES * DC_STAGE + 2 * DC_WIDTH * 4 + DC_WARPS * (DC_WIDTH / DC_CTAS) * 4;

struct DcLayer {
  const float* W;   // [in][out]
  const float* b;   // or NULL
  int in, out, act;
  int log_slice;    // outputs of a CTA, 4 .. 128, as a power of two
  int vec;          // rows of W can be read 16 bytes at a time
};
struct DcArgs {
  DcLayer layer[DC_MAX_LAYERS];
  int layers;
  const float* x;
  float* y;
  int64_t n;
};

__device__ __forceinline__ void dc_copy16(void* dst, const void* src, int bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void dc_copy4(void* dst, const void* src, int bytes) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(bytes) : "memory");
}

// NB: columns of a cluster
template <int NB>
__global__ void __launch_bounds__(DC_THREADS, 1) dense_chain_kernel(const __grid_constant__ DcArgs A) {
  fb_after_previous();
  extern __shared__ __align__(16) uint8_t dc_smem[];
  __shared__ float bias[DC_MAX_LAYERS][DC_MAX_SLICE];               // this CTA's slices
  __shared__ __align__(16) float sent[DC_WIDTH / DC_CTAS];
  float* ring = (float*)dc_smem;                                    // [stage][rows][slice]
  float* hbuf = (float*)(dc_smem + DC_STAGES * DC_STAGE);           // [2][width][NB]
  float* red = hbuf + 2 * DC_WIDTH;                                 // [warp][4][NB][slice / 4]
  uint32_t rank;
  asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
  const int64_t s0 = (int64_t)(blockIdx.x / DC_CTAS) * NB;
  const int cols = (int)(A.n - s0 < NB ? A.n - s0 : NB);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");   // (waited for below: this CTA's memory may be written to)

  // the ring's next stage: rows [pr, pr + rows) of layer pl
  int pl = 0, pr = 0, put = 0;
  auto load_next = [&]() {
    while (pl < A.layers && ((int)rank << A.layer[pl].log_slice) >= A.layer[pl].out) ++pl;   // (no outputs of this layer here)
    if (pl < A.layers) {
      const DcLayer& L = A.layer[pl];
      const int ls = L.log_slice, out = L.out, rows = min((DC_STAGE / 4) >> ls, L.in - pr), j0 = (int)rank << ls;
      float* dst = ring + put * (DC_STAGE / 4);
      const float* src = L.W + (int64_t)pr * out + j0;
      if (L.vec) {
        const int c = 4 * (tid & ((1 << (ls - 2)) - 1)), bytes = j0 + c < out ? 16 : 0;
        for (int r = tid >> (ls - 2); r < rows; r += DC_THREADS >> (ls - 2)) dc_copy16(dst + (r << ls) + c, bytes ? src + (int64_t)r * out + c : src, bytes);
      } else {
        const int c = tid & ((1 << ls) - 1), bytes = j0 + c < out ? 4 : 0;
        for (int r = tid >> ls; r < rows; r += DC_THREADS >> ls) dc_copy4(dst + (r << ls) + c, bytes ? src + (int64_t)r * out + c : src, bytes);
      }
      put = put + 1 == DC_STAGES ? 0 : put + 1;
      pr += rows;
      if (pr == L.in) {
        pr = 0;
        ++pl;
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
#pragma unroll 1
  for (int s = 0; s < DC_STAGES - 1; ++s) load_next();

  const int in0 = A.layer[0].in;
#pragma unroll 4
  for (int i = tid; i < NB * in0; i += DC_THREADS) {   // (the columns of x are neighbours in memory)
    const int n = NB == 1 ? 0 : i / in0, k = NB == 1 ? i : i - n * in0;
    hbuf[k * NB + n] = n < cols ? __ldg(A.x + s0 * in0 + i) : 0.0f;
  }
  if (tid < DC_MAX_SLICE)
    for (int l = 0; l < A.layers; ++l) {
      const int j = ((int)rank << A.layer[l].log_slice) + tid;
      bias[l][tid] = tid < (1 << A.layer[l].log_slice) && j < A.layer[l].out && A.layer[l].b != nullptr ? __ldg(A.layer[l].b + j) : 0.0f;
    }
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  int get = 0;
#pragma unroll 1
  for (int l = 0; l < A.layers; ++l) {
    const DcLayer& L = A.layer[l];
    const int ls = L.log_slice, out = L.out, in = L.in, act = L.act, j0 = (int)rank << ls, cgs = 1 << (ls - 2);
    const bool last = l + 1 == A.layers;
    const float* h = hbuf + (l & 1) * DC_WIDTH;
    if (j0 < out) {
      // a lane: four outputs (lane mod cgs), rows of its own
      const int cg = lane & (cgs - 1), r0 = (warp << (7 - ls)) + (lane >> (ls - 2)), step = DC_WARPS << (7 - ls);
      float acc[NB][4];
#pragma unroll
      for (int n = 0; n < NB; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[n][e] = 0.0f;
#pragma unroll 1
      for (int k0 = 0; k0 < in;) {
        asm volatile("cp.async.wait_group %0;" ::"n"(DC_STAGES - 2) : "memory");
        __syncthreads();   // the stage is there for all, and the one before has been read by all
        load_next();
        const int rows = min((DC_STAGE / 4) >> ls, in - k0);
        const float* w = ring + get * (DC_STAGE / 4) + 4 * cg;
        const float* hk = h + k0 * NB;
#pragma unroll 4
        for (int r = r0; r < rows; r += step) {
          const float4 v = *(const float4*)(w + (r << ls));
          float x[NB];
          if (NB >= 4) {
#pragma unroll
            for (int n = 0; n < NB; n += 4) *(float4*)(x + n) = *(const float4*)(hk + r * NB + n);
          } else {
#pragma unroll
            for (int n = 0; n < NB; ++n) x[n] = hk[r * NB + n];
          }
#pragma unroll
          for (int n = 0; n < NB; ++n) {
            acc[n][0] = fmaf(v.x, x[n], acc[n][0]);
            acc[n][1] = fmaf(v.y, x[n], acc[n][1]);
            acc[n][2] = fmaf(v.z, x[n], acc[n][2]);
            acc[n][3] = fmaf(v.w, x[n], acc[n][3]);
          }
        }
        k0 += rows;
        get = get + 1 == DC_STAGES ? 0 : get + 1;
      }
      // over the lanes that share outputs, then over the warps
      for (int o = cgs; o < 32; o *= 2)
#pragma unroll
        for (int n = 0; n < NB; ++n)
#pragma unroll
          for (int e = 0; e < 4; ++e) acc[n][e] += __shfl_xor_sync(0xffffffffu, acc[n][e], o);
      const int outs = NB << ls;
      if (lane < cgs)
#pragma unroll
        for (int n = 0; n < NB; ++n)
#pragma unroll
          for (int e = 0; e < 4; ++e) red[warp * outs + ((e * NB + n) << (ls - 2)) + cg] = acc[n][e];
      __syncthreads();
      if (tid < outs) {
        float s = 0.0f;
#pragma unroll
        for (int w = 0; w < DC_WARPS; ++w) s += red[w * outs + tid];
        const int en = tid >> (ls - 2), n = en % NB, jl = 4 * (tid & (cgs - 1)) + en / NB, j = j0 + jl;
        s = fb_act_apply(act, s + bias[l][jl]);
        if (!last) sent[jl * NB + n] = s;
        else if (j < out && n < cols) A.y[(s0 + n) * out + j] = s;
      }
      if (!last) {
        // warp w sends the slice to CTA w, in 16-byte pieces (word by word to all CTAs the pushes took 2 us a layer)
        __syncthreads();
        const uint32_t next = (uint32_t)__cvta_generic_to_shared(hbuf + ((l + 1) & 1) * DC_WIDTH + j0 * NB);
        uint32_t peer;
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(peer) : "r"(next), "r"(warp));
        for (int i = 4 * lane; i < outs && j0 * NB + i < out * NB; i += 128) {
          const float4 v = *(const float4*)(sent + i);
          asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(peer + 4u * (uint32_t)i), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w) : "memory");
        }
      }
    }
    if (!last) {
      asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
      asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    }
  }
}

template <int NB>
int32_t launch(fb_ctx* ctx, cudaStream_t stream, const DcArgs& A) {
  cudaLaunchConfig_t lc = {};
  cudaLaunchAttribute at[2];
  at[1] = fb_early_start();
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = DC_CTAS;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  lc.gridDim = dim3((unsigned)((A.n + NB - 1) / NB * DC_CTAS));
  lc.blockDim = dim3(DC_THREADS);
  lc.dynamicSmemBytes = DC_SMEM;
  lc.stream = stream;
  lc.attrs = at;
  lc.numAttrs = 2;
  FB_ONCE(ctx, FB_CUDA(fb_allow_smem(dense_chain_kernel<NB>, DC_SMEM)); FB_CUDA(cudaFuncSetAttribute(dense_chain_kernel<NB>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1)));
  FB_CUDA(cudaLaunchKernelEx(&lc, dense_chain_kernel<NB>, A));
  FB_LAUNCH_CHECK();
  return FB_OK;
}

}  // namespace

// How many clusters are resident at once (7 on a whole B200: the largest GPCs hold one each; called by fb_ctx_create).
void fb_dense_chain_query_clusters(fb_ctx* ctx) {
  cudaLaunchConfig_t lc = {};
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = DC_CTAS;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  lc.gridDim = dim3(DC_CTAS);
  lc.blockDim = dim3(DC_THREADS);
  lc.dynamicSmemBytes = DC_SMEM;
  lc.attrs = at;
  lc.numAttrs = 1;
  int n = 0;
  if (fb_allow_smem(dense_chain_kernel<4>, DC_SMEM) != cudaSuccess ||
      cudaFuncSetAttribute(dense_chain_kernel<4>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess ||
      cudaOccupancyMaxActiveClusters(&n, dense_chain_kernel<4>, &lc) != cudaSuccess) {
    cudaGetLastError();
    n = 0;
  }
  ctx->chain_clusters = n;
}

FB_API int32_t fb_dense_chain_fwd(fb_ctx* ctx, void* stream, const int64_t* table, int32_t layers, const float* x, float* y, int64_t n) {
  FB_CHECK_CTX(ctx);
  FB_REQUIRE(table && x && y, FB_ERR_INVALID_ARG, "fb_dense_chain_fwd: NULL pointer");
  if (layers < 2 || layers > DC_MAX_LAYERS || n < 1) return FB_ERR_UNSUPPORTED;
  DcArgs A;
  A.layers = layers; A.x = x; A.y = y; A.n = n;
  int64_t bytes = 0, widest = 0;
  for (int l = 0; l < layers; ++l) {
    const int64_t* t = table + 5 * l;   // W, b, in, out, activation
    const int64_t in = t[2], out = t[3];
    FB_REQUIRE(t[0] != 0 && fb_act_valid((int)t[4]) && (l == 0 || in == A.layer[l - 1].out), FB_ERR_INVALID_ARG, "fb_dense_chain_fwd: bad layer %d", l);
    if (in < 1 || out < 1 || in > DC_WIDTH || out > DC_CTAS * DC_MAX_SLICE) return FB_ERR_UNSUPPORTED;
    DcLayer& L = A.layer[l];
    L.W = (const float*)t[0]; L.b = (const float*)t[1]; L.in = (int)in; L.out = (int)out; L.act = (int)t[4];
    L.log_slice = 2;
    while ((DC_CTAS << L.log_slice) < out) ++L.log_slice;
    L.vec = (out % 4 == 0 && fb_aligned16(L.W)) ? 1 : 0;
    bytes += 4 * in * out;
    widest = in > widest ? in : widest;
    if (l + 1 < layers && out > widest) widest = out;
  }
  // As many columns in a cluster as its buffers hold, up to 4: with 8 the sums cost more device time than a layer's launch (512 -> 512:
  // 5.1 us a layer against 4.6; 3.8 with 4, 3.3 with 1).
  int nb = n >= 3 ? 4 : (int)n;
  while (nb > 1 && widest * nb > DC_WIDTH) nb /= 2;
  for (int l = 0; l < layers; ++l)
    while (nb > 1 && (nb << A.layer[l].log_slice) > DC_WIDTH / DC_CTAS) nb /= 2;
  // Weights through 16 SMs instead of all: from about 2 MB a layer on (1.25 with 3 or 4 columns) the layers alone are faster (1024 -> 1024,
  // 4 MB: 9 us a layer here, 7 alone), and a second wave of clusters would double the time.
  if (bytes > layers * (nb <= 2 ? (int64_t)2 << 20 : (int64_t)5 << 18) || (n + nb - 1) / nb > ctx->chain_clusters) return FB_ERR_UNSUPPORTED;
  switch (nb) {
    case 4: return launch<4>(ctx, (cudaStream_t)stream, A);
    case 2: return launch<2>(ctx, (cudaStream_t)stream, A);
    default: return launch<1>(ctx, (cudaStream_t)stream, A);
  }
}
