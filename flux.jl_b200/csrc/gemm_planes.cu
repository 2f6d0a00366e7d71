// Tensor-core GEMM for Float32 data as products of two half-precision planes per operand (planes.cu): A_lo B_hi + A_hi B_lo +
// A_hi B_hi by tcgen05.mma.kind::f16, which multiplies at twice the TF32 rate of the 3xTF32 kernel (gemm_tc.cu).
//
// Tiles: 256 x 256 of a CTA pair (cta_group::2: each CTA holds 128 rows of A and 128 columns of B) or 128 x 128 of one CTA, k-blocks
// of 64: one image of each operand and stage, 64 KB, three stages.  The kernel is persistent and schedules as the 3xTF32
// kernel does (gemm_sched.cuh): whole tiles with stride G, a last wave cut along K, or (SPLIT) one wave of tiles whose K range
// is shared by a cluster.
//
// Sums.  The tensor core adds into its Float32 accumulator with truncation, 3.5e-9 of the result's norm per k-value of one
// accumulation (half of 3xTF32: an MMA takes 16 k-values here).  K is cut into segments of 512 that alternate between two
// accumulator buffers, and the epilogue warps add each finished one to sums in registers, to nearest, while the MMAs fill the
// other: eight warps hold a 128 x 256 half tile (128 sums a thread).  Error 1.8e-6 of the result's norm whatever K is (3xTF32:
// 1.5e-5 at K >= 2048).  8192 x 4096 x 4096 with the operands' split, without left-out elements: 584 us; segments of 256 608 us
// (9.3e-7), of 128 635 us; through C, as the 3xTF32 kernel does it, 764 us with segments of 2048.
//
// Elements that the images leave out (planes.cu) are added to the same sums in Float32, from the operands themselves, while the MMAs work
// on the next segment: some 2 us a chunk of 32 x 32 sums that has any.  A row with more of them than its list holds sets a word: this
// kernel then does nothing, and the 3xTF32 kernel behind it, which otherwise finds nothing to do (4 us), makes the product.
//
// Stores go through 4 KB of shared memory a warp, so that eight lanes write one 128-byte line; with a row per lane (16 bytes of
// 32 lines at a time) products of K = 1024 were bound by their stores (16384 x 1024 x 1024 without left-out elements: 174 -> 121 us).
//
// Bound: tensor pipe under the power limit: 8192 x 4096 x 4096 without the split 537 us = 1536 TFLOP/s issued, 0.90 of the measured
// rate of a plain bf16 product (1711 TFLOP/s).  3xTF32, with the split in the kernel: 1048 us.
//
// Warp 0 issues the TMA loads, warp 1 owns tensor memory and issues the MMAs, warps 2-9 are the epilogue: warp w reads the TMEM lane
// quadrant w % 4 and one half of the columns.  No TMA load is multicast.  Every wait is bounded: error codes 1201 / 1202.
#include <cuda.h>

#include "common.cuh"
#include "gemm_sched.cuh"
#include "tc_common.cuh"

namespace {

constexpr int BM = 128;
constexpr int HBK = 64;                       // k-values per k-block (128 bytes of each plane)
constexpr int PLANE_BYTES = BM * HBK * 2, IMG_BYTES = 2 * PLANE_BYTES;
constexpr int STAGE_BYTES = 2 * IMG_BYTES, STAGES = 3;
constexpr int OUT_OFFSET = STAGES * STAGE_BYTES, OUT_BYTES = 8 * 4096;   // eight warps' store buffers
constexpr int BAR_OFFSET = OUT_OFFSET + OUT_BYTES;
constexpr int SMEM_BYTES = BAR_OFFSET + 512 + 1024;   // barriers + alignment slack
constexpr int EPI_WARPS = 8, NUM_THREADS = 32 * (2 + EPI_WARPS);
constexpr int UNIT_KB = 8;                    // k-blocks of a unit of the tail split
constexpr int SEG_KB = 8;                     // k-blocks of an accumulation segment

// v * 2^e for |e| <= 252, in two factors that are normal numbers: halfway between v and the result neither overflows where the
// result does not
__device__ __forceinline__ float unscale(float v, int e) {
  const int h = e >> 1;
  return v * __int_as_float((h + 127) << 23) * __int_as_float((e - h + 127) << 23);
}
// One lane issues, its operands moved to uniform registers one by one (the other GEMM kernels' way takes 88 -> 64 clocks an MMA): here the quicker issue
// makes the kernel slower, alone as well as at the power limit (8192 x 4096 x 4096: 533 us so, 542 by a converged warp, each within 1 us over
// several runs in turn; what it then waits for was not found).
template <bool PAIR>
__device__ __forceinline__ void tc_mma_h(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  if (PAIR)
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, {%5, %5, %5, %5, %5, %5, %5, %5}, p;\n\t}"
        ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate), "r"(0u)
        : "memory");
  else
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %5, %5, %5}, p;\n\t}"
        ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate), "r"(0u)
        : "memory");
}
__device__ __forceinline__ void commit_own(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void commit_pair(uint32_t bar, uint16_t mask) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar), "h"(mask) : "memory");
}

// One operand as its elements are read beside its images: those that the images leave out are listed row by row (planes.cu)
struct Side {
  const float* X;
  int64_t ld;
  int mn_major;
  const int32_t *exps, *left;
  const int2* list;
  __device__ __forceinline__ float at(int row, int k) const { return __ldg(X + (mn_major ? (int64_t)k * ld + row : (int64_t)row * ld + k)); }
};
struct Out {
  float* C;
  int64_t ldc;
  float* Z;
  const float* bias;
  const int32_t *ea, *eb;
  int M, N, act, accumulate;
  Side a, b;
  int cap;
  float least;            // the scaled magnitude from which on the images hold an element
  const int32_t* over;   // set: a row has more such elements than its list holds, 3xTF32 makes this product
};

__device__ __forceinline__ float scale_of(const Side& s, int row) { return __int_as_float((127 - __ldg(s.exps + row)) << 23); }
// the listed element of a row with the smallest k behind `last`: (k, bits of the scaled element)
__device__ __forceinline__ int2 next_left(const Side& s, int row, int count, int cap, int last) {
  const int2* list = s.list + (int64_t)row * cap;
  int2 best = __ldg(list);
  if (count == 1) return best;
  best.x = 0x7fffffff;
  for (int i = 0; i < count; ++i) {
    const int2 e = __ldg(list + i);
    if (e.x > last && e.x < best.x) best = e;
  }
  return best;
}
// Adds what the images leave out of 32 rows x 32 columns to `sums` (scaled; a row is eight float4, exchanged as below), in Float32 and in
// one order: the c-th elements of the rows, then those of the columns times the elements of A that its image holds, for c = 0, 1, ...
// rl, cl: how many the lane's row and column have.  Eight loads are in flight at a time.  Not inlined: its registers are not the caller's.
__device__ __noinline__ void add_left_out(const Out& o, float* sums, int row0, int col0, int rl, int cl) {
  const int lane = threadIdx.x & 31, row = row0 + lane, col = col0 + lane;
  const float sa = row < o.M ? scale_of(o.a, row) : 0.0f, sb = col < o.N ? scale_of(o.b, col) : 0.0f;
  auto sum = [&](int r, int c) -> float& { return sums[(r * 8 + ((c >> 2) ^ (r & 7))) * 4 + (c & 3)]; };
  const int most = __reduce_max_sync(0xffffffffu, max(rl, cl));
  int2 ea = make_int2(-1, 0), eb = make_int2(-1, 0);
  for (int c = 0; c < most; ++c) {
    if (c < rl) ea = next_left(o.a, row, rl, o.cap, ea.x);
    if (c < cl) eb = next_left(o.b, col, cl, o.cap, eb.x);
    __syncwarp();
    uint32_t rows = __ballot_sync(0xffffffffu, c < rl), cols = __ballot_sync(0xffffffffu, c < cl);
    while (rows != 0) {
      int r[8];
      float v[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        r[u] = __ffs(rows) - 1;
        rows &= rows - 1;
        const int k = __shfl_sync(0xffffffffu, ea.x, r[u] & 31);
        v[u] = r[u] >= 0 && col < o.N ? o.b.at(col, k) : 0.0f;
      }
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const float x = __int_as_float(__shfl_sync(0xffffffffu, ea.y, r[u] & 31));
        if (r[u] >= 0) sum(r[u], lane) = fmaf(x, v[u] * sb, sum(r[u], lane));
      }
    }
    __syncwarp();
    while (cols != 0) {
      int q[8];
      float v[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        q[u] = __ffs(cols) - 1;
        cols &= cols - 1;
        const int k = __shfl_sync(0xffffffffu, eb.x, q[u] & 31);
        v[u] = q[u] >= 0 && row < o.M ? o.a.at(row, k) : 0.0f;
      }
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const float y = __int_as_float(__shfl_sync(0xffffffffu, eb.y, q[u] & 31));
        if (q[u] >= 0 && !fb_planes_leaves_out(v[u], sa, o.least)) sum(lane, q[u]) = fmaf(v[u] * sa, y, sum(lane, q[u]));
      }
    }
    __syncwarp();
  }
}
// columns n .. n + 3 of one row, complete: undo the operands' scales, add C, bias, pre-activation store, activation, store
__device__ __forceinline__ void emit4(const Out& o, int row, int n, float4 u, int er, const int4& ec, const float4& b4) {
  if (row >= o.M || n >= o.N) return;
  u.x = unscale(u.x, er + ec.x); u.y = unscale(u.y, er + ec.y); u.z = unscale(u.z, er + ec.z); u.w = unscale(u.w, er + ec.w);
  float* c = o.C + (int64_t)row * o.ldc + n;
  float* z = o.Z ? o.Z + (int64_t)row * o.ldc + n : nullptr;
  if (n + 3 < o.N) {
    if (o.accumulate) {
      const float4 c4 = *(const float4*)c;
      u.x += c4.x; u.y += c4.y; u.z += c4.z; u.w += c4.w;
    }
    u.x += b4.x; u.y += b4.y; u.z += b4.z; u.w += b4.w;
    if (z) *(float4*)z = u;
    if (o.act != FB_ACT_IDENTITY) {
      u.x = fb_act_apply(o.act, u.x); u.y = fb_act_apply(o.act, u.y); u.z = fb_act_apply(o.act, u.z); u.w = fb_act_apply(o.act, u.w);
    }
    *(float4*)c = u;
  } else {
    const float t[4] = {u.x, u.y, u.z, u.w}, b[4] = {b4.x, b4.y, b4.z, b4.w};
#pragma unroll
    for (int e = 0; e < 3; ++e) {
      if (n + e >= o.N) break;
      float x = t[e];
      if (o.accumulate) x += c[e];
      x += b[e];
      if (z) z[e] = x;
      c[e] = fb_act_apply(o.act, x);
    }
  }
}
// the column exponents and biases of columns n .. n + 3 (zero where there is none)
__device__ __forceinline__ void load_cols(const Out& o, int n, int4& ec, float4& b4) {
  ec = make_int4(0, 0, 0, 0);
  b4 = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  if (n >= o.N) return;
  ec = __ldg((const int4*)(o.eb + n));   // padded to whole tiles
  if (o.bias == nullptr) return;
  if (n + 3 < o.N) {
    b4 = __ldg((const float4*)(o.bias + n));
  } else {
    b4.x = __ldg(o.bias + n);
    if (n + 1 < o.N) b4.y = __ldg(o.bias + n + 1);
    if (n + 2 < o.N) b4.z = __ldg(o.bias + n + 2);
  }
}

template <bool PAIR, bool SPLIT>
__global__ void __launch_bounds__(NUM_THREADS, 1)
gemm_planes_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const __grid_constant__ Out out, int K,
                   int32_t* __restrict__ dev_err, int a_mn, int b_mn, const Sched sch) {
  fb_after_previous();
  constexpr int BN = PAIR ? 256 : 128;
  constexpr int TMEM_COLS = 2 * BN;                 // two accumulator buffers
  constexpr int RANKS = PAIR ? 2 : 1;
  constexpr int NC = BN / 64;                       // chunks of 32 columns of one epilogue warp
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  const uint32_t smem_base = smem_u32(smem);
  uint64_t* bars = (uint64_t*)(smem + BAR_OFFSET);
  const uint32_t bar_base = smem_base + BAR_OFFSET;
  // barrier slots: full[S], empty[S], tmem_full[2], tmem_empty[2]
  auto full_bar = [&](int s) { return bar_base + 8u * (uint32_t)s; };
  auto empty_bar = [&](int s) { return bar_base + 8u * (uint32_t)(STAGES + s); };
  auto tmem_full_bar = [&](int b) { return bar_base + 8u * (uint32_t)(2 * STAGES + b); };
  auto tmem_empty_bar = [&](int b) { return bar_base + 8u * (uint32_t)(2 * STAGES + 2 + b); };
  volatile uint32_t* s_tmem = (volatile uint32_t*)(bars + 2 * STAGES + 4);
  volatile int* s_abort = (volatile int*)(bars + 2 * STAGES + 5);
  volatile int* s_skip = (volatile int*)(bars + 2 * STAGES + 6);   // [0] mine, [1] written by the cluster's first CTA

  const int warp = uniform_warp(), lane = threadIdx.x & 31;
  const int ksplit = SPLIT ? sch.ksplit : 1;
  const uint32_t crank = (PAIR || SPLIT) ? cluster_ctarank() : 0u;
  const uint32_t rank = PAIR ? (crank & 1u) : 0u;   // half of the pair's tile
  const uint32_t lead_rank = crank - rank;
  const bool leader = (rank == 0);
  const int cid = PAIR ? (int)(blockIdx.x >> 1) : (int)blockIdx.x;
  const int G = PAIR ? (int)(gridDim.x >> 1) : (int)gridDim.x;
  const int num_kb = (K + HBK - 1) / HBK;
  // first row of A / C and first column of B this CTA loads in tile t, and the tile's first column
  auto tile_m0 = [&](int t) { return (t / sch.tiles_n) * (BM * RANKS) + BM * (int)rank; };
  auto tile_n0 = [&](int t) { return (t % sch.tiles_n) * BN; };

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(full_bar(s), 1);
      mbar_init(empty_bar(s), 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(tmem_full_bar(b), 1);
      mbar_init(tmem_empty_bar(b), EPI_WARPS * RANKS);
    }
    *s_abort = 0;
    // an error word left set means: do not start; 3xTF32 makes products of rows with too much left out
    s_skip[0] = (*(volatile int32_t*)dev_err != 0 || *out.over != 0) ? 1 : 0;
    s_skip[1] = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    fence_proxy_async();
  }
  if (PAIR || SPLIT) {
    __syncwarp();
    cluster_sync_all();   // all CTAs of the cluster run and their barriers exist: remote accesses may start
    if (threadIdx.x == 0 && crank == 0) {
      // the whole cluster must take the same decision: its first CTA's
      for (uint32_t r = 0; r < (uint32_t)(ksplit * RANKS); ++r)
        asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(map_to_cta(smem_u32((const void*)(s_skip + 1)), r)), "r"((int)s_skip[0])
                     : "memory");
    }
    __syncwarp();
    cluster_sync_all();
    if (s_skip[1] != 0) return;
  } else {
    __syncthreads();
    if (s_skip[0] != 0) return;
  }

  if (warp == 1) {
    if (PAIR) {
      asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32((const void*)s_tmem)),
                   "r"((uint32_t)TMEM_COLS)
                   : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    } else {
      asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32((const void*)s_tmem)),
                   "r"((uint32_t)TMEM_COLS)
                   : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = __reduce_or_sync(0xffffffffu, *s_tmem);

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer ---
    if (lane == 0) {
      int it = 0;   // k-blocks issued so far over all tiles: names the stage and its phase
      bool ok = true;
      WorkIter<SPLIT, UNIT_KB> wi(sch, cid, G);
      Portion p;
      while (ok && wi.next(sch, cid, G, num_kb, p)) {
        const int ia = tile_m0(p.tile) / BM * num_kb, ib = (tile_n0(p.tile) / BM + (int)rank) * num_kb;   // first images
        for (int kb = p.kb0; kb < p.kb1; ++kb, ++it) {
          const int s = it % STAGES;
          const uint32_t ph = (uint32_t)(it / STAGES) & 1u;
          ok = mbar_wait_cluster(empty_bar(s), ph ^ 1u, s_abort);
          if (!ok) break;
          // pairs: the leader's barrier counts the bytes of both CTAs; the peer only issues its loads
          const uint32_t fb = PAIR ? map_to_cta(full_bar(s), lead_rank) : full_bar(s);
          if (leader) mbar_arrive_expect_tx(full_bar(s), (uint32_t)(RANKS * STAGE_BYTES));
          const uint32_t dst = smem_base + (uint32_t)(s * STAGE_BYTES);
          if (PAIR) {
            tma_load_2d_pair(dst, &tmA, 0, (ia + kb) * (2 * BM), fb);
            tma_load_2d_pair(dst + (uint32_t)IMG_BYTES, &tmB, 0, (ib + kb) * (2 * BM), fb);
          } else {
            tma_load_2d(dst, &tmA, 0, (ia + kb) * (2 * BM), fb);
            tma_load_2d(dst + (uint32_t)IMG_BYTES, &tmB, 0, (ib + kb) * (2 * BM), fb);
          }
        }
      }
    }
  } else if (warp == 1) {
    // -------------------------------------------------- MMA issuer (the leader CTA of a pair) ---
    if (lane == 0 && leader) {
      // instruction descriptor: D = F32, A = B = F16 (code 0), operand majors, N >> 3, M >> 4
      const uint32_t idesc = (1u << 4) | ((uint32_t)a_mn << 15) | ((uint32_t)b_mn << 16) | ((uint32_t)(BN >> 3) << 17) |
                             ((uint32_t)((BM * RANKS) >> 4) << 24);
      // image descriptors: the high word (version 1, 128-byte swizzle, 8-row atoms) is one constant; the low word holds the address
      // and the stride between MN-major chunks.  A k-step is 32 bytes of a K-major row or sixteen 128-byte rows of an MN-major chunk
      const uint64_t high = (uint64_t)((2u << 29) | (1u << 14) | (1024u >> 4)) << 32;
      const uint32_t a_lbo = (a_mn ? (uint32_t)(HBK * 128 >> 4) : 1u) << 16, b_lbo = (b_mn ? (uint32_t)(HBK * 128 >> 4) : 1u) << 16;
      const uint32_t a_step = a_mn ? 2048u >> 4 : 32u >> 4, b_step = b_mn ? 2048u >> 4 : 32u >> 4;
      bool ok = true;
      int it = 0, sc = 0;   // k-blocks and accumulation segments issued so far over all tiles
      WorkIter<SPLIT, UNIT_KB> wi(sch, cid, G);
      Portion p;
      while (ok && wi.next(sch, cid, G, num_kb, p))
        for (int kb = p.kb0, kb_in_seg = 0; kb < p.kb1 && ok; ++kb, ++it) {
          const int s = it % STAGES;
          const uint32_t ph = (uint32_t)(it / STAGES) & 1u;
          const int buf = sc & 1, use = sc >> 1;
          if (kb_in_seg == 0 && use > 0) {
            // the epilogue warps must have drained this accumulator buffer's previous segment
            ok = mbar_wait_cluster(tmem_empty_bar(buf), (uint32_t)(use - 1) & 1u, s_abort);
            if (!ok) break;
          }
          ok = mbar_wait_cluster(full_bar(s), ph, s_abort);
          if (!ok) break;
          tc_fence_after();
          const uint32_t d_tmem = tmem_base + (uint32_t)(buf * BN);
          const uint32_t a_s = smem_base + (uint32_t)(s * STAGE_BYTES);
          const uint32_t al0 = ((a_s >> 4) & 0x3fffu) | a_lbo, bl0 = (((a_s + (uint32_t)IMG_BYTES) >> 4) & 0x3fffu) | b_lbo;
          constexpr uint32_t LO = (uint32_t)PLANE_BYTES >> 4;   // from the upper plane to the lower one
#pragma unroll
          for (int kk = 0; kk < HBK / 16; ++kk) {
            const uint32_t al = al0 + (uint32_t)kk * a_step, bl = bl0 + (uint32_t)kk * b_step;
            tc_mma_h<PAIR>(d_tmem, high | (al + LO), high | bl, idesc, (kb_in_seg > 0 || kk > 0) ? 1u : 0u);
            tc_mma_h<PAIR>(d_tmem, high | al, high | (bl + LO), idesc, 1u);
            tc_mma_h<PAIR>(d_tmem, high | al, high | bl, idesc, 1u);
          }
          const bool seg_end = (kb_in_seg == SEG_KB - 1 || kb == p.kb1 - 1);
          if (PAIR) {
            commit_pair(empty_bar(s), (uint16_t)(3u << lead_rank));                 // frees the stage in both CTAs
            if (seg_end) commit_pair(tmem_full_bar(buf), (uint16_t)(3u << lead_rank));
          } else {
            commit_own(empty_bar(s));
            if (seg_end) commit_own(tmem_full_bar(buf));
          }
          kb_in_seg = seg_end ? 0 : kb_in_seg + 1;
          if (seg_end) ++sc;
        }
    }
  } else {
    // -------------------------------------------------------------- epilogue warps ---
    const int q = warp & 3, half = (warp - 2) >> 2;
    const int trow = 32 * q + lane;               // this lane's row of the CTA's 128
    float4* stage = (float4*)(smem + OUT_OFFSET) + (warp - 2) * 256;
    bool ok = true;
    int sc = 0;                                   // segments drained so far over all tiles
    WorkIter<SPLIT, UNIT_KB> wi(sch, cid, G);
    Portion p;
    while (ok && wi.next(sch, cid, G, num_kb, p)) {
      const int m0 = tile_m0(p.tile), n0 = tile_n0(p.tile) + half * (BN / 2);
      // A part of a split tile collects its sums in a workspace slot: [column quad][row] float4.  The parts of a tile are the
      // CTAs c_first .. c_last whose unit ranges meet it (those with an empty range excepted).
      int c_first = 0, c_last = 0, nparts = 0, rem_first = 0, r_first = 0, u_lo = 0;
      int* ticket = nullptr;
      const int step_q = sch.U / G, step_r = sch.U % G;
      auto slot = [&](int pc, int trail) {
        return (float4*)sch.ws + (size_t)((2 * pc + trail) * RANKS + (int)rank) * (BM * 64) + half * (BN / 8) * BM + trow;
      };
      // f(part, trail) for every part of the tile in k order; r(pc) = floor(pc * U / G), the first unit of CTA pc, is stepped
      // without dividing
      auto each_part = [&](auto f) {
        int r0 = r_first, rem = rem_first;
        for (int pc = c_first; pc <= c_last; ++pc) {
          int r1 = r0 + step_q, rem1 = rem + step_r;
          if (rem1 >= G) { rem1 -= G; ++r1; }
          if (r1 > r0) f(pc, r0 < u_lo ? 1 : 0);
          r0 = r1;
          rem = rem1;
        }
      };
      if (!SPLIT && p.partial) {
        u_lo = p.tail_tile * sch.nu;
        const int u_hi = u_lo + sch.nu - 1;
        c_first = (int)(((long long)(u_lo + 1) * G - 1) / sch.U);
        c_last = (int)(((long long)(u_hi + 1) * G - 1) / sch.U);
        ticket = sch.tickets + (c_first * RANKS + (int)rank) * EPI_WARPS + (warp - 2);
        r_first = (int)((long long)c_first * sch.U / G);
        rem_first = (int)((long long)c_first * sch.U % G);
        each_part([&](int, int) { ++nparts; });
      }
      // columns 32 cc .. 32 cc + 31 of the warp's rows, one row a lane, to C: eight lanes share a row's 128 bytes
      const int r0 = m0 + 32 * q + (lane >> 3);
      const int ea_lane = m0 + trow < out.M ? __ldg(out.ea + m0 + trow) : 0;
      const bool plain = out.act == FB_ACT_IDENTITY && out.Z == nullptr && !out.accumulate;
      auto store = [&](const float* v, int cc) {
#pragma unroll
        for (int j = 0; j < 8; ++j) stage[lane * 8 + (j ^ (lane & 7))] = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
        __syncwarp();
        const int n = n0 + 32 * cc + 4 * (lane & 7);
        int4 ec;
        float4 b4;
        load_cols(out, n, ec, b4);
        if (plain && n0 + 32 * cc + 31 < out.N) {
          float* c = out.C + (int64_t)r0 * out.ldc + n;
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const int r = 4 * i + (lane >> 3);
            float4 u = stage[r * 8 + ((lane & 7) ^ (r & 7))];
            const int er = __shfl_sync(0xffffffffu, ea_lane, r);
            u.x = unscale(u.x, er + ec.x) + b4.x; u.y = unscale(u.y, er + ec.y) + b4.y;
            u.z = unscale(u.z, er + ec.z) + b4.z; u.w = unscale(u.w, er + ec.w) + b4.w;
            if (r0 + 4 * i < out.M) *(float4*)(c + (int64_t)(4 * i) * out.ldc) = u;
          }
        } else {
#pragma unroll 2
          for (int i = 0; i < 8; ++i) {
            const int r = 4 * i + (lane >> 3);
            emit4(out, m0 + 32 * q + r, n, stage[r * 8 + ((lane & 7) ^ (r & 7))], __shfl_sync(0xffffffffu, ea_lane, r), ec, b4);
          }
        }
        __syncwarp();
      };
      const int nseg = (p.kb1 - p.kb0 + SEG_KB - 1) / SEG_KB;
      float sum[NC][32];
#pragma unroll
      for (int cc = 0; cc < NC; ++cc)
#pragma unroll
        for (int i = 0; i < 32; ++i) sum[cc][i] = 0.0f;
      bool fused = false;
      // What the images leave out belongs to the part with the first k-values: a chunk of 32 columns behind each of its segments, while the
      // MMAs work on the next.  (Behind the last segment, in the store: 8192 x 4096 x 4096 took 606 - 644 us.)
      const bool first_part = p.kb0 == 0;
      int rl = 0, cl[NC];     // how many elements, of the lane's row and of its column of each chunk
      if (first_part) rl = m0 + trow < out.M ? __ldg(out.a.left + m0 + trow) : 0;
#pragma unroll
      for (int cc = 0; cc < NC; ++cc) cl[cc] = first_part && n0 + 32 * cc + lane < out.N ? __ldg(out.b.left + n0 + 32 * cc + lane) : 0;
      auto left_out = [&](int cc, int cl_cc, float (&to)[32]) {
        if (!__any_sync(0xffffffffu, (rl | cl_cc) != 0)) return;
#pragma unroll
        for (int j = 0; j < 8; ++j) stage[lane * 8 + j] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        __syncwarp();
        add_left_out(out, (float*)stage, m0 + 32 * q, n0 + 32 * cc, rl, cl_cc);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float4 x = stage[lane * 8 + (j ^ (lane & 7))];
          to[4 * j] += x.x; to[4 * j + 1] += x.y; to[4 * j + 2] += x.z; to[4 * j + 3] += x.w;
        }
        __syncwarp();
      };
      for (int seg = 0; seg < nseg && ok; ++seg, ++sc) {
        const int buf = sc & 1, use = sc >> 1;
        ok = mbar_wait_cluster(tmem_full_bar(buf), (uint32_t)use & 1u, s_abort);
        if (!ok) break;
        tc_fence_after();
        const uint32_t acc = tmem_base + ((uint32_t)(32 * q) << 16) + (uint32_t)(buf * BN + half * (BN / 2));
#pragma unroll
        for (int cc = 0; cc < NC; ++cc) {
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            uint32_t r[16];
            tc_ld_32x32b_x16(acc + (uint32_t)(32 * cc + 16 * h), r);
            tc_wait_ld();
#pragma unroll
            for (int i = 0; i < 16; ++i) sum[cc][16 * h + i] += __uint_as_float(r[i]);
          }
        }
        // this buffer may be overwritten once every epilogue warp (of both CTAs) has read its part
        tc_fence_before();
        __syncwarp();
        if (lane == 0) {
          if (PAIR) mbar_arrive_cluster(map_to_cta(tmem_empty_bar(buf), lead_rank));
          else mbar_arrive(tmem_empty_bar(buf));
        }
#pragma unroll
        for (int cc = 0; cc < NC; ++cc)
          if (cc == seg || (seg == nseg - 1 && cc > seg)) left_out(cc, cl[cc], sum[cc]);
      }
      if (!ok) break;
      if (!SPLIT && p.partial && cid == c_first) {
        // The first part of a tile usually finishes last (it is the end of its CTA's range, the other parts are the beginning
        // of theirs).  When every other part has already drawn its ticket, their slots are complete: add them on the way out.
        int seen = 0;
        if (lane == 0) seen = *(volatile int*)ticket;
        seen = __shfl_sync(0xffffffffu, seen, 0);
        fused = (seen == nparts - 1);
        if (fused) __threadfence();
      }
#pragma unroll
      for (int cc = 0; cc < NC; ++cc) {
        if (n0 + 32 * cc >= out.N) break;   // warp-uniform
        float(&v)[32] = sum[cc];
        if (SPLIT) {
          // the sums go to shared memory (all MMAs have read their stages by now), from where the cluster adds them up
          float4* d4 = (float4*)((float*)smem + trow * (BN + 4) + half * (BN / 2) + cc * 32);
#pragma unroll
          for (int j = 0; j < 8; ++j) d4[j] = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
        } else if (!p.partial) {
          store(v, cc);
        } else if (fused) {
          each_part([&](int pc, int trail) {
            if (pc == c_first) return;
            const float4* s4 = slot(pc, trail) + 8 * cc * BM;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              const float4 x = __ldcg(s4 + j * BM);
              v[4 * j] += x.x; v[4 * j + 1] += x.y; v[4 * j + 2] += x.z; v[4 * j + 3] += x.w;
            }
          });
          store(v, cc);
        } else {
          float4* s4 = slot(cid, p.trail) + 8 * cc * BM;
#pragma unroll
          for (int j = 0; j < 8; ++j) s4[j * BM] = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
        }
      }
      if (!SPLIT && p.partial && !fused) {
        // whoever draws the last ticket adds the slots up, in k order (the same sums as the fused path makes)
        __threadfence();
        __syncwarp();
        int drawn = 0;
        if (lane == 0) drawn = atomicAdd(ticket, 1);
        drawn = __shfl_sync(0xffffffffu, drawn, 0);
        if (drawn == nparts - 1) {
          __threadfence();
#pragma unroll 1
          for (int cc = 0; cc < NC; ++cc) {
            if (n0 + 32 * cc >= out.N) break;
            float v[32];
#pragma unroll
            for (int i = 0; i < 32; ++i) v[i] = 0.0f;
            each_part([&](int pc, int trail) {
              const float4* s4 = slot(pc, trail) + 8 * cc * BM;
#pragma unroll
              for (int j = 0; j < 8; ++j) {
                const float4 x = __ldcg(s4 + j * BM);
                v[4 * j] += x.x; v[4 * j + 1] += x.y; v[4 * j + 2] += x.z; v[4 * j + 3] += x.w;
              }
            });
            store(v, cc);
          }
        }
      }
    }
  }

  // ---------------------------------------------- split K: the cluster adds up its parts ---
  if (SPLIT) {
    __syncwarp();
    cluster_sync_all();
    const int part = cid % ksplit, rows = BM / ksplit;
    const int m0 = tile_m0(cid / ksplit), n0 = tile_n0(cid / ksplit);
    for (int e = threadIdx.x; e < rows * (BN / 4); e += NUM_THREADS) {
      const int r = part * rows + e / (BN / 4), c = 4 * (e % (BN / 4));
      if (m0 + r >= out.M || n0 + c >= out.N) continue;
      const uint32_t src = smem_base + (uint32_t)((r * (BN + 4) + c) * 4);
      float4 x[8];
#pragma unroll
      for (int i = 0; i < 8; ++i)
        if (i < ksplit) {
          const uint32_t a = map_to_cta(src, (uint32_t)(i * RANKS) + rank);
          asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(x[i].x), "=f"(x[i].y), "=f"(x[i].z), "=f"(x[i].w) : "r"(a) : "memory");
        }
      float4 v = x[0];
#pragma unroll
      for (int i = 1; i < 8; ++i)
        if (i < ksplit) { v.x += x[i].x; v.y += x[i].y; v.z += x[i].z; v.w += x[i].w; }
      int4 ec;
      float4 b4;
      load_cols(out, n0 + c, ec, b4);
      emit4(out, m0 + r, n0 + c, v, __ldg(out.ea + m0 + r), ec, b4);
    }
  }

  // ---------------------------------------------------------------------- teardown ---
  tc_fence_before();
  __syncthreads();
  if (PAIR || SPLIT) cluster_sync_all();   // no CTA may release its tensor or shared memory while a peer can still touch it
  if (warp == 1) {
    __syncwarp();
    if (PAIR)
      asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"((uint32_t)TMEM_COLS) : "memory");
    else
      asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"((uint32_t)TMEM_COLS) : "memory");
  }
  if (threadIdx.x == 0 && *s_abort != 0) atomicExch(dev_err, PAIR ? 1202 : 1201);
}

// --------------------------------------------------------------------------- host side ---
// images as rows of 128 bytes; one box is an image
bool encode_map_img(CUtensorMap* map, const uint16_t* img, int64_t rows) {
  EncodeTiledFn fn = get_encode_fn();
  if (!fn) return false;
  cuuint64_t gdim[2] = {(cuuint64_t)HBK, (cuuint64_t)rows};
  cuuint64_t gstride[1] = {(cuuint64_t)HBK * 2};
  cuuint32_t box[2] = {(cuuint32_t)HBK, 2 * BM};
  cuuint32_t estr[2] = {1, 1};
  return fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, (void*)img, gdim, gstride, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
            CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

struct Plan {
  double time;      // modelled, us
  bool pair;        // 256 x 256 tiles of a CTA pair, else 128 x 128 of one CTA
  int ksplit;       // CTAs (pairs) of a cluster that share a tile
  bool tail;        // the last wave is cut along K and dealt out over all CTAs
};

template <bool PAIR, bool SPLIT>
int32_t launch(fb_ctx* ctx, cudaStream_t stream, const fb_gemm_args& a, const Plan& plan) {
  constexpr int BN = PAIR ? 256 : 128, RANKS = PAIR ? 2 : 1;
  const int64_t tiles_n = (a.N + BN - 1) / BN, num_tiles = (a.M + BM * RANKS - 1) / (BM * RANKS) * tiles_n;
  const int sms = ctx->sm_count - ctx->reserved_sms;
  const int64_t Gmax = sms / RANKS > 0 ? sms / RANKS : 1;
  const int num_kb = (int)((a.K + HBK - 1) / HBK);
  Sched sch;
  sch.num_tiles = (int)num_tiles;
  sch.tiles_n = (int)tiles_n;
  sch.dp_tiles = (int)num_tiles;
  sch.nu = (num_kb + UNIT_KB - 1) / UNIT_KB;
  sch.U = 0;
  sch.ksplit = plan.ksplit;
  sch.seg = 0;             // (SEG_KB, a constant of the kernel)
  sch.run_if = nullptr;
  sch.ws = nullptr;
  sch.tickets = nullptr;
  int64_t G = SPLIT ? num_tiles * plan.ksplit : Gmax < num_tiles ? Gmax : num_tiles;
  const int64_t rest = num_tiles % Gmax;
  const bool tail = !SPLIT && plan.tail && rest * sch.nu < 0x40000000;
  // tickets of the parts of a tail, what else starts at zero, images, slots for the parts (two per CTA)
  const size_t image_bytes = fb_planes_bytes(a);
  const size_t tickets = tail ? ((size_t)(Gmax * RANKS) * EPI_WARPS * sizeof(int) + 255) / 256 * 256 : 0;
  const size_t slots = tail ? (size_t)BM * 256 * sizeof(float) * 2 * (size_t)(Gmax * RANKS) : 0;
  const fb_temp mem(ctx, stream, tickets + image_bytes + slots);
  if (mem.p == nullptr) return FB_ERR_UNSUPPORTED;
  FB_CUDA(cudaMemsetAsync(mem.p, 0, tickets + fb_planes_zero_bytes(a), stream));
  fb_planes planes;
  int32_t st = fb_planes_split(stream, a, (char*)mem.p + tickets, &planes);
  if (st != FB_OK) return st;
  if (tail) {
    sch.tickets = (int*)mem.p;
    sch.ws = (float*)((char*)mem.p + tickets + image_bytes);
    sch.dp_tiles = (int)(num_tiles - rest);
    sch.U = (int)(rest * sch.nu);
    G = Gmax;
  }
  CUtensorMap tmA, tmB;
  if (!encode_map_img(&tmA, planes.img[0], planes.rows[0]) || !encode_map_img(&tmB, planes.img[1], planes.rows[1]))
    return fb_fail(FB_ERR_CUDA, "gemm: cuTensorMapEncodeTiled failed (M=%lld N=%lld K=%lld)", (long long)a.M, (long long)a.N, (long long)a.K);
  auto kern = gemm_planes_kernel<PAIR, SPLIT>;
  FB_ONCE(ctx, FB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES)));
  // the whole L1 / shared array as shared memory: the communication-stream kernels ask for the same split, and an SM
  // takes CTAs of two kernels together only when their splits agree
  FB_ONCE(ctx, FB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared)));
  Out out;
  out.C = a.C; out.ldc = a.ldc; out.Z = a.Z; out.bias = a.bias_n;
  out.ea = planes.exps[0]; out.eb = planes.exps[1];
  out.M = (int)a.M; out.N = (int)a.N; out.act = a.act; out.accumulate = a.accumulate;
  out.a = {a.A, a.lda, a.a_mn_major, planes.exps[0], planes.left[0], planes.list[0]};
  out.b = {a.B, a.ldb, a.b_mn_major, planes.exps[1], planes.left[1], planes.list[1]};
  out.cap = planes.cap;
  out.least = fb_planes_least(a.K);
  out.over = planes.over;
  cudaLaunchConfig_t lc;
  memset(&lc, 0, sizeof(lc));
  lc.gridDim = dim3((unsigned)(RANKS * G), 1, 1);
  lc.blockDim = dim3(NUM_THREADS, 1, 1);
  lc.dynamicSmemBytes = SMEM_BYTES;
  lc.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[1] = fb_early_start();
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = RANKS * plan.ksplit;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  lc.attrs = attr;
  lc.numAttrs = 2;
  FB_CUDA(cudaLaunchKernelEx(&lc, kern, tmA, tmB, out, (int)a.K, ctx->dev_error, a.a_mn_major, a.b_mn_major, sch));
  FB_LAUNCH_CHECK();
  return fb_gemm_tc_launch(ctx, stream, a, 3, planes.over);
}

// The smallest modelled time (us, fitted to measurements on B200): the split kernels 3.5 each and their bytes at 6.3 TB/s, the zeroing
// before them and the 3xTF32 kernel that finds nothing to do 4.5; a k-block of 64 1.0 (pair) or 0.78 (one CTA), a tile 4 / 1.5 besides,
// 10 more (5 from K = 2048 on, behind whose segments they are hidden) for the elements that images leave out, a launch with what no other tile hides 16 / 8, a cluster's reduction 3.5,
// parts of a tail as in the 3xTF32 plan.
Plan plan_planes(const fb_ctx* ctx, const fb_gemm_args& a) {
  const int sms = ctx->sm_count - ctx->reserved_sms;
  const int num_kb = (int)((a.K + HBK - 1) / HBK);
  const double kb_bytes = (double)a.K * ((double)a.M * (a.a_mn_major ? 12 : 8) + (double)a.N * (a.b_mn_major ? 12 : 8));
  const double split = (a.a_mn_major || a.b_mn_major ? 7.0 : 3.5) + 4.5 + kb_bytes / 6.3e6;
  Plan best = {1e30, false, 1, false};
  for (int pair = 1; pair >= 0; --pair) {
    const int ranks = pair ? 2 : 1, bm = pair ? 256 : 128;
    if (pair && (a.M <= 128 || a.N <= 128)) continue;
    const double t_kb = pair ? 1.0 : 0.78, t_tile = (pair ? 4.0 : 1.5) + (num_kb < 32 ? 10.0 : 5.0), base = (pair ? 16.0 : 8.0) + split;
    const int64_t tiles = ((a.M + bm - 1) / bm) * ((a.N + bm - 1) / bm), slots = sms / ranks > 0 ? sms / ranks : 1;
    const int64_t full = tiles / slots, rest = tiles % slots;
    double t = base + full * (num_kb * t_kb + t_tile);
    bool tail = false;
    if (rest != 0) {
      const double whole = num_kb * t_kb + t_tile;
      const int64_t nu = (num_kb + UNIT_KB - 1) / UNIT_KB, units = (rest * nu + slots - 1) / slots;
      const double kb = (double)(units * UNIT_KB < num_kb ? units * UNIT_KB : num_kb);
      const double cut = nu < 2 ? 1e30 : kb * t_kb + t_tile + 12.0 + 5.0 * (double)(nu / units + 1);
      tail = cut < whole;
      t += tail ? cut : whole;
    }
    if (t < best.time) best = {t, pair != 0, 1, tail};
    for (int lg = 1; lg < 4 && ctx->reserved_sms == 0; ++lg) {
      const int s = 1 << lg;
      if (num_kb < 2 * s || s * ranks > 8 || tiles > ctx->clusters[lg + ranks - 1]) break;
      t = base + 3.5 + ((num_kb + s - 1) / s) * t_kb + t_tile;
      if (t < best.time) best = {t, pair != 0, s, false};
    }
  }
  return best;
}

}  // namespace

double fb_gemm_planes_time(const fb_ctx* ctx, const fb_gemm_args& a) { return plan_planes(ctx, a).time; }

int32_t fb_gemm_planes_launch(fb_ctx* ctx, cudaStream_t stream, const fb_gemm_args& a) {
  // Images of more than 768 MB are made piece by piece (the context's pool keeps 1 GB from call to call), cut along the longest side.
  constexpr size_t IMAGES_MAX = (size_t)768 << 20;
  if (fb_planes_bytes(a) > IMAGES_MAX && a.K >= 1024) {
    fb_gemm_args first = a, rest = a;
    if (a.K >= a.M && a.K >= a.N) {
      // the second part adds to the first one's sums and has the epilogue
      first.K = (a.K / 2 + 511) / 512 * 512;
      rest.K = a.K - first.K;
      rest.A += first.K * (a.a_mn_major ? a.lda : 1);
      rest.B += first.K * (a.b_mn_major ? a.ldb : 1);
      rest.accumulate = 1;
      first.act = FB_ACT_IDENTITY;
      first.Z = nullptr;
      first.bias_n = nullptr;
    } else if (a.M >= a.N) {
      first.M = (a.M / 2 + 255) / 256 * 256;
      rest.M = a.M - first.M;
      rest.A += first.M * (a.a_mn_major ? 1 : a.lda);
      rest.C += first.M * a.ldc;
      if (a.Z) rest.Z += first.M * a.ldc;
    } else {
      first.N = (a.N / 2 + 255) / 256 * 256;
      rest.N = a.N - first.N;
      rest.B += first.N * (a.b_mn_major ? 1 : a.ldb);
      rest.C += first.N;
      if (a.Z) rest.Z += first.N;
      if (a.bias_n) rest.bias_n += first.N;
    }
    // (once the first piece has been added to C the call has to be finished here, with 3xTF32 if memory has run out by then)
    const int32_t st = fb_gemm_planes_launch(ctx, stream, first);
    if (st != FB_OK) return st;
    const int32_t st2 = fb_gemm_planes_launch(ctx, stream, rest);
    return st2 == FB_ERR_UNSUPPORTED ? fb_gemm_tc_launch(ctx, stream, rest, 3) : st2;
  }
  const Plan p = plan_planes(ctx, a);
  if (p.pair) return p.ksplit > 1 ? launch<true, true>(ctx, stream, a, p) : launch<true, false>(ctx, stream, a, p);
  return p.ksplit > 1 ? launch<false, true>(ctx, stream, a, p) : launch<false, false>(ctx, stream, a, p);
}
