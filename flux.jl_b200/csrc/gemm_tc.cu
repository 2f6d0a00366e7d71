// Tensor-core GEMM for Float32 data on sm_100a: TMA -> shared memory -> tcgen05.mma (TF32, accumulators
// in tensor memory) -> tcgen05.ld epilogue with fused bias / activation / pre-activation store.
//
// fp32 accuracy comes from the error-compensated "3xTF32" scheme.  Operand tiles land in shared memory as raw
// fp32; the tensor core ignores the 13 low mantissa bits of a TF32 operand (measured: clearing them first gives
// bit-identical results), so the raw tile is the "hi" operand and split warps only write lo = x - trunc_tf32(x)
// beside it.  The accumulator receives A_lo*B_hi + A_hi*B_lo + A_hi*B_hi; the dropped lo*lo term is ~2^-20.
//
// Tiles.  One CTA computes a 128 x BN tile of row-major C[M][N] (BN = 256 or 128); or, for large problems, a
// cluster of two CTAs computes a 256 x 256 tile with cta_group::2 MMAs: each CTA loads and splits 128 rows of A
// and 128 columns of B, the leader CTA issues one M = 256 MMA per k-step that reads both CTAs' shared memory,
// and each CTA's tensor memory receives its own 128 rows.  K is walked in blocks of 16 floats through a ring of
// 4-7 stages.  No TMA load is multicast.
//
// The kernel is persistent: one CTA (pair) per SM (pair of SMs) walks the tile grid with stride G, the stage ring
// and the two accumulator buffers run on across tiles, so the epilogue of one tile overlaps the main loop of the
// next and barrier / tensor-memory setup is paid once per launch.
//
// Warp roles: warp 0 issues TMA loads; warp 1 owns tensor memory and issues the MMAs; warps 2-5 are the
// epilogue (one TMEM lane quadrant each); the remaining warps are groups of four split warps (two groups for the
// one-CTA tile, four for the pair) that take k-blocks in turn, so that the latency of one split (load, store,
// proxy fence, arrive) overlaps the splits of the following blocks.
//
// Operands may be K-major (k contiguous) or MN-major (m / n contiguous) in global memory; the shared-memory
// layouts are the canonical ones the MMA descriptors name: 64-byte swizzle for K-major tiles (8 rows x 64 B
// atoms) and, for MN-major tiles, the 128-byte swizzle with 32-byte atoms (128 B x 4 k-rows per atom), which
// is the only MN-major layout the tensor core accepts for 32-bit operands.
//
// The tensor core adds into its fp32 accumulator with truncation, so a long K chain drifts: the error of a sum of
// L k-values is 7.3e-9 L of the result's norm (N(0, 1) operands), whatever K is.  K is therefore cut into segments
// that alternate between two accumulator buffers in tensor memory: while the MMAs fill one, the epilogue warps
// drain the other and add it to the segments before with round-to-nearest adds (in C; a launch of one wave: in
// the CTA's slot of the workspace, where a lane's 16 bytes lie beside the next lane's: a drain of 128 x 256 then
// costs about 2.5 us, through rows of C or of the slot four to eight times that).  segment_kblocks() says how long
// a segment is.
//
// Every mbarrier wait is bounded; when a wait runs out the kernel records a code in the context's
// device error word, every role leaves its loop, tensor memory is released and the kernel returns.
#include <cuda.h>
#include <stdlib.h>

#include "common.cuh"
#include "gemm_sched.cuh"
#include "tc_common.cuh"

namespace {

constexpr int BM = 128;
constexpr int BK = 16;               // floats per k-block (64 bytes)
constexpr int UNIT_KB = 32;            // k-blocks of a unit of the tail split (gemm_sched.cuh)
constexpr int SEG_KB = 128;          // the longest accumulation segment in k-blocks (2048 k-values)

template <int BN, int PASSES, bool PAIR, int SG>
struct Cfg {
  static constexpr int SPLIT_GROUPS = SG;                   // groups of four split warps taking k-blocks in turn
  static_assert(!PAIR || PASSES == 3, "the two-CTA tile exists for the 3-pass scheme only");
  static constexpr int BNC = PAIR ? BN / 2 : BN;            // B columns this CTA loads per stage
  static constexpr int A_BYTES = BM * BK * 4;               // 8 KB
  static constexpr int B_BYTES = BNC * BK * 4;              // 16 KB at 256 columns
  static constexpr int STAGE_BYTES = (PASSES == 3 ? 2 : 1) * (A_BYTES + B_BYTES);
  static constexpr int STAGES = (229376 / STAGE_BYTES) > 8 ? 8 : (229376 / STAGE_BYTES);   // 224 KB of stages at most
  static constexpr int BAR_OFFSET = STAGES * STAGE_BYTES;
  static constexpr int SMEM_BYTES = BAR_OFFSET + 512 + 1024;   // barriers + alignment slack
  static constexpr int TMEM_COLS = 2 * BN;                  // two accumulator buffers
  static constexpr int NUM_WARPS = 6 + (PASSES == 3 ? 4 * SPLIT_GROUPS : 0);
  static constexpr int NUM_THREADS = 32 * NUM_WARPS;
  static constexpr uint32_t ARRIVALS = PAIR ? 8 : 4;        // four warps per CTA arrive on ready / tmem_empty
};

// SPLIT: a launch of one wave whose tiles are shared by the CTAs of a cluster (sch.ksplit > 1) or take several accumulation
// segments.  A kernel of its own: with both kinds in one the plain launches of small K lose 10 % (336 x 3136 x 120: 16.5
// -> 18.6 us), tiles of a pair up to 12 %.
template <bool A_MN, bool B_MN, int BN, int PASSES, bool PAIR, int SG, bool SPLIT>
__global__ void __launch_bounds__(Cfg<BN, PASSES, PAIR, SG>::NUM_THREADS, 1)
gemm_tc_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
               float* __restrict__ C, int64_t ldc, float* __restrict__ Z, const float* __restrict__ bias_n, int M,
               int N, int K, int act, int accumulate, int32_t* __restrict__ dev_err, int a3d, int b3d,
               const Sched sch) {
  fb_after_previous();
  using cfg = Cfg<BN, PASSES, PAIR, SG>;
  constexpr int SPLIT_GROUPS = SG;
  constexpr int STAGES = cfg::STAGES;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  const uint32_t smem_base = smem_u32(smem);
  uint64_t* bars = (uint64_t*)(smem + cfg::BAR_OFFSET);
  const uint32_t bar_base = smem_base + cfg::BAR_OFFSET;
  // barrier slots: full[S], ready[S], empty[S], tmem_full[2], tmem_empty[2]
  auto full_bar = [&](int s) { return bar_base + 8u * (uint32_t)s; };
  auto ready_bar = [&](int s) { return bar_base + 8u * (uint32_t)(STAGES + s); };
  auto empty_bar = [&](int s) { return bar_base + 8u * (uint32_t)(2 * STAGES + s); };
  auto tmem_full_bar = [&](int b) { return bar_base + 8u * (uint32_t)(3 * STAGES + b); };
  auto tmem_empty_bar = [&](int b) { return bar_base + 8u * (uint32_t)(3 * STAGES + 2 + b); };
  volatile uint32_t* s_tmem = (volatile uint32_t*)(bars + 3 * STAGES + 4);
  volatile int* s_abort = (volatile int*)(bars + 3 * STAGES + 5);
  volatile int* s_skip = (volatile int*)(bars + 3 * STAGES + 6);   // [0] mine, [1] written by the peer CTA

  const int warp = uniform_warp(), lane = threadIdx.x & 31;
  const bool ksplit = SPLIT && !PAIR && sch.ksplit > 1;   // (pairs take whole tiles: the spare registers of their 22 warps are few)
  const uint32_t crank = (PAIR || ksplit) ? cluster_ctarank() : 0u;
  const uint32_t rank = PAIR ? crank : 0u;   // half of the pair's tile
  const bool leader = (rank == 0);
  const int cid = PAIR ? (int)(blockIdx.x >> 1) : (int)blockIdx.x;
  const int G = PAIR ? (int)(gridDim.x >> 1) : (int)gridDim.x;
  const int tiles_n = sch.tiles_n;
  const int num_kb = (K + BK - 1) / BK;
  // rows of A / C this CTA owns in tile t, the tile's first column, and the first B column this CTA loads
  auto tile_m0 = [&](int t) { return PAIR ? (t / tiles_n) * 256 + 128 * (int)rank : (t / tiles_n) * BM; };
  auto tile_n0 = [&](int t) { return (t % tiles_n) * BN; };

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(full_bar(s), 1);
      mbar_init(ready_bar(s), cfg::ARRIVALS);
      mbar_init(empty_bar(s), 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(tmem_full_bar(b), 1);
      mbar_init(tmem_empty_bar(b), cfg::ARRIVALS);
    }
    *s_abort = 0;
    // an error word left set by an earlier launch means: do not start
    s_skip[0] = (*(volatile int32_t*)dev_err != 0 || (sch.run_if != nullptr && *sch.run_if == 0)) ? 1 : 0;
    s_skip[1] = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    fence_proxy_async();
  }
  if (PAIR || ksplit) {
    __syncwarp();
    cluster_sync_all();   // all CTAs of the cluster run and their barriers exist: remote accesses may start
    if (threadIdx.x == 0 && crank == 0) {
      // the whole cluster must take the same decision: its first CTA's
      for (uint32_t r = 0; r < (PAIR ? 2u : (uint32_t)sch.ksplit); ++r)
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
                   "r"((uint32_t)cfg::TMEM_COLS)
                   : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    } else {
      asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32((const void*)s_tmem)),
                   "r"((uint32_t)cfg::TMEM_COLS)
                   : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = __reduce_or_sync(0xffffffffu, *s_tmem);

  // u: 4 consecutive columns starting at n of one row.  add_c: add what C holds; fin: this is the tile's final value,
  // so bias, pre-activation store and activation apply.
  auto emit4 = [&](int row, float* u, int n, bool add_c, bool fin) {
    if (row >= M) return;
    float* crow = C + (int64_t)row * ldc;
    float* zrow = Z ? Z + (int64_t)row * ldc : nullptr;
    if (n + 3 < N) {
      if (add_c) {
        const float4 c4 = *(const float4*)(crow + n);
        u[0] += c4.x; u[1] += c4.y; u[2] += c4.z; u[3] += c4.w;
      }
      if (fin) {
        if (bias_n) {
          const float4 b4 = __ldg((const float4*)(bias_n + n));
          u[0] += b4.x; u[1] += b4.y; u[2] += b4.z; u[3] += b4.w;
        }
        if (zrow) *(float4*)(zrow + n) = make_float4(u[0], u[1], u[2], u[3]);
        if (act != FB_ACT_IDENTITY) {
#pragma unroll
          for (int e = 0; e < 4; ++e) u[e] = fb_act_apply(act, u[e]);
        }
      }
      *(float4*)(crow + n) = make_float4(u[0], u[1], u[2], u[3]);
    } else {
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        if (n + e >= N) break;
        float x = u[e];
        if (add_c) x += crow[n + e];
        if (fin) {
          if (bias_n) x += __ldg(bias_n + n + e);
          if (zrow) zrow[n + e] = x;
          x = fb_act_apply(act, x);
        }
        crow[n + e] = x;
      }
    }
  };

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer ---
    if (lane == 0) {
      int m0 = 0, nb0 = 0;
      int it = 0;   // k-blocks issued so far over all tiles: names the stage and its phase
      bool ok = true;
      WorkIter<SPLIT, UNIT_KB> wi(sch, cid, G);
      Portion p;
      while (ok && wi.next(sch, cid, G, num_kb, p)) {
        m0 = tile_m0(p.tile);
        nb0 = tile_n0(p.tile) + (PAIR ? cfg::BNC * (int)rank : 0);
        for (int kb = p.kb0; kb < p.kb1; ++kb, ++it) {
          const int s = it % STAGES;
          const uint32_t ph = (uint32_t)(it / STAGES) & 1u;
          ok = mbar_wait_cluster(empty_bar(s), ph ^ 1u, s_abort);
          if (!ok) break;
          mbar_arrive_expect_tx(full_bar(s), (uint32_t)(cfg::A_BYTES + cfg::B_BYTES));
          const uint32_t a_dst = smem_base + (uint32_t)(s * cfg::STAGE_BYTES);
          const uint32_t b_dst = a_dst + (uint32_t)((PASSES == 3 ? 2 : 1) * cfg::A_BYTES);
          const int k0 = kb * BK;
          if (A_MN) {
            if (a3d) {
              tma_load_3d(a_dst, &tmA, 0, k0, m0 >> 5, full_bar(s));
            } else {
#pragma unroll
              for (int c = 0; c < BM / 32; ++c) tma_load_2d(a_dst + (uint32_t)(c * BK * 128), &tmA, m0 + 32 * c, k0, full_bar(s));
            }
          } else {
            tma_load_2d(a_dst, &tmA, k0, m0, full_bar(s));
          }
          if (B_MN) {
            if (b3d) {
              tma_load_3d(b_dst, &tmB, 0, k0, nb0 >> 5, full_bar(s));
            } else {
#pragma unroll
              for (int c = 0; c < cfg::BNC / 32; ++c) tma_load_2d(b_dst + (uint32_t)(c * BK * 128), &tmB, nb0 + 32 * c, k0, full_bar(s));
            }
          } else {
            tma_load_2d(b_dst, &tmB, k0, nb0, full_bar(s));
          }
        }
      }
    }
  } else if (warp == 1) {
    // -------------------------------------------------- MMA issuer (the leader CTA of a pair) ---
    if (leader) {
      // instruction descriptor: D = F32, A = B = TF32, operand majors, N >> 3, M >> 4
      const uint32_t idesc = (1u << 4) | (2u << 7) | (2u << 10) | ((A_MN ? 1u : 0u) << 15) | ((B_MN ? 1u : 0u) << 16) |
                             ((uint32_t)(BN >> 3) << 17) | ((uint32_t)((PAIR ? 256 : BM) >> 4) << 24);
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
          ok = warp_wait_cluster(tmem_empty_bar(buf), (uint32_t)(use - 1) & 1u, s_abort);
          if (!ok) break;
        }
        ok = warp_wait_cluster(PASSES == 3 ? ready_bar(s) : full_bar(s), ph, s_abort);
        if (!ok) break;
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + (uint32_t)(buf * BN);
        const uint32_t a_hi = smem_base + (uint32_t)(s * cfg::STAGE_BYTES);
        const uint32_t a_lo = a_hi + (uint32_t)cfg::A_BYTES;
        const uint32_t b_hi = a_hi + (uint32_t)((PASSES == 3 ? 2 : 1) * cfg::A_BYTES);
        const uint32_t b_lo = b_hi + (uint32_t)cfg::B_BYTES;
#pragma unroll
        for (int kk = 0; kk < BK / 8; ++kk) {
          // one MMA covers 8 k-values: 32 bytes along a K-major row, eight 128-byte k-rows of an MN-major tile
          const uint32_t a_off = A_MN ? (uint32_t)(kk * 1024) : (uint32_t)(kk * 32);
          const uint32_t b_off = B_MN ? (uint32_t)(kk * 1024) : (uint32_t)(kk * 32);
          const uint64_t da_hi = A_MN ? make_smem_desc(a_hi + a_off, BK * 128, 512, LAYOUT_SW128_32B)
                                      : make_smem_desc(a_hi + a_off, 16, 512, LAYOUT_SW64);
          const uint64_t db_hi = B_MN ? make_smem_desc(b_hi + b_off, BK * 128, 512, LAYOUT_SW128_32B)
                                      : make_smem_desc(b_hi + b_off, 16, 512, LAYOUT_SW64);
          const uint32_t first = (kb_in_seg > 0 || kk > 0) ? 1u : 0u;
          if (PASSES == 3) {
            const uint64_t da_lo = A_MN ? make_smem_desc(a_lo + a_off, BK * 128, 512, LAYOUT_SW128_32B)
                                        : make_smem_desc(a_lo + a_off, 16, 512, LAYOUT_SW64);
            const uint64_t db_lo = B_MN ? make_smem_desc(b_lo + b_off, BK * 128, 512, LAYOUT_SW128_32B)
                                        : make_smem_desc(b_lo + b_off, 16, 512, LAYOUT_SW64);
            if (PAIR) {
              tc_mma2_tf32(d_tmem, da_lo, db_hi, idesc, first);
              tc_mma2_tf32(d_tmem, da_hi, db_lo, idesc, 1u);
              tc_mma2_tf32(d_tmem, da_hi, db_hi, idesc, 1u);
            } else {
              tc_mma_tf32(d_tmem, da_lo, db_hi, idesc, first);
              tc_mma_tf32(d_tmem, da_hi, db_lo, idesc, 1u);
              tc_mma_tf32(d_tmem, da_hi, db_hi, idesc, 1u);
            }
          } else {
            tc_mma_tf32(d_tmem, da_hi, db_hi, idesc, first);
          }
        }
        const bool seg_end = (kb_in_seg == sch.seg - 1 || kb == p.kb1 - 1);
        if (PAIR) {
          tc_commit2_mc(empty_bar(s), (uint16_t)3);                 // frees the stage in both CTAs
          if (seg_end) tc_commit2_mc(tmem_full_bar(buf), (uint16_t)3);
        } else {
          tc_commit(empty_bar(s));
          if (seg_end) tc_commit(tmem_full_bar(buf));
        }
        kb_in_seg = seg_end ? 0 : kb_in_seg + 1;
        if (seg_end) ++sc;
      }
    }
  } else if (warp < 6) {
    // -------------------------------------------------------------- epilogue warps ---
    const int q = warp & 3;                 // TMEM lane quadrant this warp may read
    constexpr int RANKS = PAIR ? 2 : 1;
    bool ok = true;
    int sc = 0;                             // segments drained so far over all tiles
    WorkIter<SPLIT, UNIT_KB> wi(sch, cid, G);
    Portion p;
    while (ok && wi.next(sch, cid, G, num_kb, p)) {
      const int n0 = tile_n0(p.tile);
      const int row = tile_m0(p.tile) + 32 * q + lane;
      // A part of a split tile collects its sums in a workspace slot (always 256 floats per row).  The parts of
      // a tile are the CTAs c_first .. c_last whose unit ranges meet it (those with an empty range excepted).
      float* srow = nullptr;
      int c_first = 0, c_last = 0, nparts = 0, rem_first = 0, r_first = 0, u_lo = 0;
      int* ticket = nullptr;
      const int row_off = (32 * q + lane) * 256;
      const int step_q = sch.U / G, step_r = sch.U % G;
      // where earlier segments wait: the warp's 16-byte pieces of one column quad lie side by side
      float4* park = SPLIT ? (float4*)(sch.ws + (size_t)blockIdx.x * BM * 256) + 32 * q + lane : nullptr;
      if (!SPLIT && p.partial) {
        srow = sch.ws + (size_t)((2 * cid + p.trail) * RANKS + (int)rank) * BM * 256 + row_off;
        u_lo = p.tail_tile * sch.nu;
        const int u_hi = u_lo + sch.nu - 1;
        c_first = (int)(((long long)(u_lo + 1) * G - 1) / sch.U);
        c_last = (int)(((long long)(u_hi + 1) * G - 1) / sch.U);
        ticket = sch.tickets + (c_first * RANKS + (int)rank) * 4 + q;
        // r(pc) = floor(pc * U / G), the first unit of CTA pc, is stepped from c_first on without dividing
        r_first = (int)((long long)c_first * sch.U / G);
        rem_first = (int)((long long)c_first * sch.U % G);
        int r0 = r_first;
        int rem = rem_first;
        for (int pc = c_first; pc <= c_last; ++pc) {
          int r1 = r0 + step_q;
          int rem1 = rem + step_r;
          if (rem1 >= G) { rem1 -= G; ++r1; }
          nparts += (r1 > r0) ? 1 : 0;
          r0 = r1;
          rem = rem1;
        }
      }
      // v[0 .. 4 * NV) += columns [col, col + 4 * NV) of this lane's row summed over parts pc_from .. c_last, in order
      auto add_parts = [&](float* v, int col, int pc_from) {
        int r0 = r_first;
        int rem = rem_first;
        for (int pc = c_first; pc <= c_last; ++pc) {
          int r1 = r0 + step_q;
          int rem1 = rem + step_r;
          if (rem1 >= G) { rem1 -= G; ++r1; }
          if (r1 > r0 && pc >= pc_from) {
            const int tr = (r0 < u_lo) ? 1 : 0;
            const float4* prow =
                (const float4*)(sch.ws + (size_t)((2 * pc + tr) * RANKS + (int)rank) * BM * 256 + row_off + col);
            float4 x[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) x[j] = __ldcg(prow + j);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              v[4 * j] += x[j].x; v[4 * j + 1] += x[j].y; v[4 * j + 2] += x[j].z; v[4 * j + 3] += x[j].w;
            }
          }
          r0 = r1;
          rem = rem1;
        }
      };
      const int nseg = (p.kb1 - p.kb0 + sch.seg - 1) / sch.seg;
      bool fused = false;
      for (int seg = 0; seg < nseg && ok; ++seg, ++sc) {
        const int buf = sc & 1, use = sc >> 1;
        ok = mbar_wait_cluster(tmem_full_bar(buf), (uint32_t)use & 1u, s_abort);
        if (!ok) break;
        tc_fence_after();
        // later segments add into what the earlier ones left (round-to-nearest fp32 adds)
        const bool last = (seg == nseg - 1);
        if (!SPLIT && p.partial && last && cid == c_first) {
          // The first part of a tile usually finishes last (it is the end of its CTA's range, the other parts are
          // the beginning of theirs).  When every other part has already drawn its ticket, their slots are
          // complete: add them to this last segment on its way out and write C directly.
          int seen = 0;
          if (lane == 0) seen = *(volatile int*)ticket;
          seen = __shfl_sync(0xffffffffu, seen, 0);
          fused = (seen == nparts - 1);
          if (fused) __threadfence();
        }
#pragma unroll 1
        for (int cc = 0; cc < BN / 32; ++cc) {
          const int nb = n0 + cc * 32;
          if (nb >= N) break;   // warp-uniform
          uint32_t r[32];
          tc_ld_32x32b_x32(tmem_base + ((uint32_t)(32 * q) << 16) + (uint32_t)(buf * BN + cc * 32), r);
          tc_wait_ld();
          float* v = reinterpret_cast<float*>(r);
          if (SPLIT || !p.partial) {
            if (SPLIT && seg > 0) {
#pragma unroll
              for (int j = 0; j < 8; ++j) {
                const float4 o = park[(8 * cc + j) * BM];
                v[4 * j] += o.x; v[4 * j + 1] += o.y; v[4 * j + 2] += o.z; v[4 * j + 3] += o.w;
              }
            }
            if (SPLIT && !last) {
#pragma unroll
              for (int j = 0; j < 8; ++j) park[(8 * cc + j) * BM] = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
            } else if (ksplit) {
              // the sums go to shared memory (all MMAs have read their stages by now), from where the cluster adds them up
              float4* d4 = (float4*)((float*)smem + (32 * q + lane) * (BN + 4) + cc * 32);
#pragma unroll
              for (int j = 0; j < 8; ++j) d4[j] = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
            } else {
              const bool add_c = (!SPLIT && seg > 0) || (accumulate != 0);
#pragma unroll
              for (int j = 0; j < 8; ++j) emit4(row, v + 4 * j, nb + 4 * j, add_c, last);
            }
          } else {
            float4* s4 = (float4*)(srow + cc * 32);
            if (seg > 0) {
#pragma unroll
              for (int j = 0; j < 8; ++j) {
                const float4 o = s4[j];
                v[4 * j] += o.x; v[4 * j + 1] += o.y; v[4 * j + 2] += o.z; v[4 * j + 3] += o.w;
              }
            }
            if (last && fused) {
              add_parts(v, cc * 32, c_first + 1);
              add_parts(v + 16, cc * 32 + 16, c_first + 1);
#pragma unroll
              for (int j = 0; j < 8; ++j) emit4(row, v + 4 * j, nb + 4 * j, accumulate != 0, true);
            } else {
#pragma unroll
              for (int j = 0; j < 8; ++j) s4[j] = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
            }
          }
        }
        // this buffer may be overwritten once every epilogue warp (of both CTAs) has read its quadrant
        tc_fence_before();
        __syncwarp();
        if (lane == 0) {
          if (PAIR) mbar_arrive_cluster(map_to_cta(tmem_empty_bar(buf), 0u));
          else mbar_arrive(tmem_empty_bar(buf));
        }
      }
      if (!SPLIT && p.partial && ok) {
        if (!fused) {
          // whoever draws the last ticket adds the slots up, in k order (the same sums as the fused path makes)
          __threadfence();
          __syncwarp();
          int drawn = 0;
          if (lane == 0) drawn = atomicAdd(ticket, 1);
          drawn = __shfl_sync(0xffffffffu, drawn, 0);
          if (drawn == nparts - 1) {
            __threadfence();
#pragma unroll 1
            for (int hc = 0; hc < BN / 16; ++hc) {
              const int nb = n0 + hc * 16;
              if (nb >= N) break;
              float v[16];
#pragma unroll
              for (int j = 0; j < 16; ++j) v[j] = 0.0f;
              add_parts(v, hc * 16, c_first);
#pragma unroll
              for (int j = 0; j < 4; ++j) emit4(row, v + 4 * j, nb + 4 * j, accumulate != 0, true);
            }
          }
        }
      }
    }
  } else {
    // ------------------------------------------- split warps: write lo = x - trunc_tf32(x) ---
    const int group = (warp - 6) >> 2;
    const int tt = ((warp - 6) & 3) * 32 + lane;   // 0..127 inside the group
    bool ok = true;
    int total_kb = 0;   // the stage ring runs on across tiles
    {
      WorkIter<SPLIT, UNIT_KB> wi(sch, cid, G);
      Portion p;
      while (wi.next(sch, cid, G, num_kb, p)) total_kb += p.kb1 - p.kb0;
    }
    for (int kb = group; kb < total_kb && ok; kb += SPLIT_GROUPS) {
      const int s = kb % STAGES;
      const uint32_t ph = (uint32_t)(kb / STAGES) & 1u;
      ok = mbar_wait(full_bar(s), ph, s_abort);
      if (!ok) break;
      const float4* a_hi = (const float4*)(smem + s * cfg::STAGE_BYTES);
      float4* a_lo = (float4*)(smem + s * cfg::STAGE_BYTES + cfg::A_BYTES);
      const float4* b_hi = (const float4*)(smem + s * cfg::STAGE_BYTES + 2 * cfg::A_BYTES);
      float4* b_lo = (float4*)(smem + s * cfg::STAGE_BYTES + 2 * cfg::A_BYTES + cfg::B_BYTES);
      constexpr int NA = cfg::A_BYTES / 16 / 128, NB = cfg::B_BYTES / 16 / 128;
      float4 v[NA + NB];
#pragma unroll
      for (int i = 0; i < NA; ++i) v[i] = a_hi[tt + i * 128];
#pragma unroll
      for (int i = 0; i < NB; ++i) v[NA + i] = b_hi[tt + i * 128];
#pragma unroll
      for (int i = 0; i < NA + NB; ++i) {
        v[i].x = tf32_lo(v[i].x); v[i].y = tf32_lo(v[i].y); v[i].z = tf32_lo(v[i].z); v[i].w = tf32_lo(v[i].w);
      }
#pragma unroll
      for (int i = 0; i < NA; ++i) a_lo[tt + i * 128] = v[i];
#pragma unroll
      for (int i = 0; i < NB; ++i) b_lo[tt + i * 128] = v[NA + i];
      fence_proxy_async();   // generic-proxy writes become visible to the tensor core's async-proxy reads
      __syncwarp();
      if (lane == 0) {
        if (PAIR) mbar_arrive_cluster(map_to_cta(ready_bar(s), 0u));
        else mbar_arrive(ready_bar(s));
      }
    }
  }

  // ---------------------------------------------- split K: the cluster adds up its parts ---
  if (ksplit) {
    __syncwarp();
    cluster_sync_all();
    const int S = sch.ksplit, part = (int)crank, rows = BM / S;
    const int m0 = tile_m0(cid / S), n0 = tile_n0(cid / S);
    for (int e = threadIdx.x; e < rows * (BN / 4); e += cfg::NUM_THREADS) {
      const int r = part * rows + e / (BN / 4), c = 4 * (e % (BN / 4));
      if (m0 + r >= M || n0 + c >= N) continue;
      const uint32_t src = smem_base + (uint32_t)((r * (BN + 4) + c) * 4);
      float4 x[8];
#pragma unroll
      for (int i = 0; i < 8; ++i)
        if (i < S) {
          const uint32_t a = map_to_cta(src, (uint32_t)i);
          asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(x[i].x), "=f"(x[i].y), "=f"(x[i].z), "=f"(x[i].w) : "r"(a) : "memory");
        }
      float v[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
      for (int i = 0; i < 8; ++i)
        if (i < S) { v[0] += x[i].x; v[1] += x[i].y; v[2] += x[i].z; v[3] += x[i].w; }
      emit4(m0 + r, v, n0 + c, accumulate != 0, true);
    }
  }

  // ---------------------------------------------------------------------- teardown ---
  tc_fence_before();
  __syncthreads();
  if (PAIR || ksplit) cluster_sync_all();   // no CTA may release its tensor or shared memory while a peer can still touch it
  if (warp == 1) {
    __syncwarp();
    if (PAIR)
      asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"((uint32_t)cfg::TMEM_COLS) : "memory");
    else
      asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"((uint32_t)cfg::TMEM_COLS) : "memory");
  }
  if (threadIdx.x == 0 && *s_abort != 0) atomicExch(dev_err, PAIR ? 1002 : 1001);
}

// --------------------------------------------------------------------------- host side ---
// Workspace of the split-tile schedule, owned by the context: slots for partial sums and the tickets.
struct Plan {
  double time;              // modelled, us
  int shape, ksplit, seg;   // tile shape (0, 1, 2: see plan_3xtf32), CTAs that share a tile, k-blocks per accumulation segment
  bool split;               // the SPLIT kernel: one wave of shared tiles, or of tiles of several segments
  bool tail;                // the last wave is cut along K and dealt out over all CTAs
  const int32_t* run_if = nullptr;   // (device) the kernel does nothing unless it is set
};

// Accumulation segment of a launch of one wave.  An even cut of all k-blocks over the SMs gives each of them num_kb * tiles / SMs
// (tiles: 256 x 256 by two SMs, 128 x 256 or 128 x 128, the largest that occupy half of the GPU); no truncating sum is longer
// than that, nor than 1664 k-values, and where the tiles fill 3/4 of the SMs by themselves 2048: a shared tile is then at
// least as exact as the tail split below would make it (104 x 1032 x 12256: 6.4e-6 of the result's norm).  Against one
// segment for every CTA's range, up to 2048: 104 x 1032 x 12256 1.1e-5 in 62 us -> 4.0e-6 in 63, 1296 x 2216 x 1528 1.1e-5
// -> 5.8e-6, both 76 us, 1024 x 1024 x 16384 1.5e-5 in 170 us -> 1.0e-5 in 163.
int segment_kblocks(const fb_gemm_args& a, int num_kb, int part_kb, int sms, int* drains) {
  const int64_t pairs = ((a.M + 255) / 256) * ((a.N + 255) / 256);
  const int64_t t256 = ((a.M + BM - 1) / BM) * ((a.N + 255) / 256), t128 = ((a.M + BM - 1) / BM) * ((a.N + 127) / 128);
  const int64_t tiles = a.M >= 256 && a.N >= 256 && 4 * pairs >= sms ? 2 * pairs : a.N <= 128 || 2 * t256 <= sms ? t128 : t256;
  int64_t most = SEG_KB;
  if (4 * tiles < 3 * (int64_t)sms) {
    most = (int64_t)num_kb * tiles / sms;
    most = most < UNIT_KB ? UNIT_KB : most > 104 ? 104 : most;
  }
  const int n = (int)((part_kb + most - 1) / most);
  *drains = n - 1;
  return (part_kb + n - 1) / n;
}

// 3-d view {32, K, MN / 32} of an MN-major matrix (row k holds MN contiguous floats): box {32, BK, chunks}.
// Only for MN a multiple of 32, so that no chunk straddles the end of a row.
bool encode_map_mn3d(CUtensorMap* map, const float* base, int64_t K, int64_t MN, int64_t ld, uint32_t chunks) {
  EncodeTiledFn fn = get_encode_fn();
  if (!fn || MN % 32 != 0) return false;
  cuuint64_t gdim[3] = {32, (cuuint64_t)K, (cuuint64_t)(MN / 32)};
  cuuint64_t gstride[2] = {(cuuint64_t)ld * sizeof(float), 128};
  cuuint32_t box[3] = {32, (cuuint32_t)BK, chunks};
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, (void*)base, gdim, gstride, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                  CU_TENSOR_MAP_SWIZZLE_128B_ATOM_32B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS;
}

template <bool A_MN, bool B_MN, int BN, int PASSES, bool PAIR, int SG, bool SPLIT>
int32_t launch_variant(fb_ctx* ctx, cudaStream_t stream, const fb_gemm_args& a, const Plan& plan) {
  using cfg = Cfg<BN, PASSES, PAIR, SG>;
  CUtensorMap tmA, tmB;
  bool ok;
  int a3d = 0, b3d = 0;
  if (A_MN) {
    a3d = encode_map_mn3d(&tmA, a.A, a.K, a.M, a.lda, BM / 32) ? 1 : 0;
    ok = a3d || encode_map(&tmA, a.A, a.K, a.M, a.lda, 32, BK, CU_TENSOR_MAP_SWIZZLE_128B_ATOM_32B);
  } else {
    ok = encode_map(&tmA, a.A, a.M, a.K, a.lda, BK, BM, CU_TENSOR_MAP_SWIZZLE_64B);
  }
  if (ok) {
    if (B_MN) {
      b3d = encode_map_mn3d(&tmB, a.B, a.K, a.N, a.ldb, cfg::BNC / 32) ? 1 : 0;
      ok = b3d || encode_map(&tmB, a.B, a.K, a.N, a.ldb, 32, BK, CU_TENSOR_MAP_SWIZZLE_128B_ATOM_32B);
    } else {
      ok = encode_map(&tmB, a.B, a.N, a.K, a.ldb, BK, cfg::BNC, CU_TENSOR_MAP_SWIZZLE_64B);
    }
  }
  if (!ok) return fb_fail(FB_ERR_CUDA, "gemm: cuTensorMapEncodeTiled failed (M=%lld N=%lld K=%lld lda=%lld ldb=%lld)",
                          (long long)a.M, (long long)a.N, (long long)a.K, (long long)a.lda, (long long)a.ldb);
  auto kern = gemm_tc_kernel<A_MN, B_MN, BN, PASSES, PAIR, SG, SPLIT>;
  FB_ONCE(ctx, FB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, cfg::SMEM_BYTES)));
  // the whole L1 / shared array as shared memory: the communication-stream kernels ask for the same split, and an SM
  // takes CTAs of two kernels together only when their splits agree
  FB_ONCE(ctx, FB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared)));
  const int tiles_n = (int)((a.N + BN - 1) / BN);
  const int64_t tiles_m = PAIR ? (a.M + 255) / 256 : (a.M + BM - 1) / BM;
  const int64_t num_tiles = tiles_m * tiles_n;
  if (num_tiles > 0x7fffffff) return fb_fail(FB_ERR_UNSUPPORTED, "gemm: too many tiles");
  // one CTA (pair) per SM (pair of SMs)
  // (fewer when the caller reserved SMs for communication kernels that run beside this one: a persistent grid that
  // does not fit waits for them to finish)
  const int sms = ctx->sm_count - ctx->reserved_sms;
  const int64_t Gmax = PAIR ? (sms / 2 > 0 ? sms / 2 : 1) : sms;
  const int num_kb = (int)((a.K + BK - 1) / BK);
  Sched sch;
  sch.num_tiles = (int)num_tiles;
  sch.tiles_n = tiles_n;
  sch.dp_tiles = (int)num_tiles;
  sch.nu = (num_kb + UNIT_KB - 1) / UNIT_KB;
  sch.U = 0;
  sch.ksplit = plan.ksplit;
  sch.seg = plan.seg;
  sch.run_if = plan.run_if;
  sch.ws = nullptr;
  sch.tickets = nullptr;
  int64_t G = Gmax < num_tiles ? Gmax : num_tiles;
  const int64_t rest = num_tiles % Gmax;
  const bool tail = !SPLIT && plan.tail && rest * sch.nu < 0x40000000;
  if (SPLIT) G = num_tiles * plan.ksplit;
  // slots for segments that wait (one per CTA), or for the parts of a tail (two per CTA, and the tickets)
  constexpr size_t SLOT = (size_t)BM * 256 * sizeof(float);
  const size_t tickets = (size_t)ctx->sm_count * 4 * sizeof(int);
  const size_t need = SPLIT ? ((num_kb + plan.ksplit - 1) / plan.ksplit > plan.seg ? SLOT * (size_t)(G * (PAIR ? 2 : 1)) : 0)
                            : tail ? SLOT * 2 * (size_t)(Gmax * (PAIR ? 2 : 1)) + tickets : 0;
  const fb_temp ws(ctx, stream, need);
  sch.ws = (float*)ws.p;
  if (need != 0 && ws.p == nullptr) {
    // no memory: whole tiles, whose segments meet in C
    if (SPLIT) return launch_variant<A_MN, B_MN, BN, PASSES, PAIR, SG, false>(ctx, stream, a, {plan.time, plan.shape, 1, plan.seg, false, false, plan.run_if});
  } else if (tail) {
    sch.dp_tiles = (int)(num_tiles - rest);
    sch.U = (int)(rest * sch.nu);
    sch.tickets = (int*)((char*)ws.p + need - tickets);
    FB_CUDA(cudaMemsetAsync(sch.tickets, 0, tickets, stream));
    G = Gmax;
  }
  cudaLaunchConfig_t lc;
  memset(&lc, 0, sizeof(lc));
  lc.gridDim = dim3((unsigned)(PAIR ? 2 * G : G), 1, 1);
  lc.blockDim = dim3(cfg::NUM_THREADS, 1, 1);
  lc.dynamicSmemBytes = cfg::SMEM_BYTES;
  lc.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[1] = fb_early_start();
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (PAIR ? 2 : 1) * plan.ksplit;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  lc.attrs = attr;
  lc.numAttrs = 2;
  FB_CUDA(cudaLaunchKernelEx(&lc, kern, tmA, tmB, a.C, a.ldc, a.Z, a.bias_n, (int)a.M, (int)a.N, (int)a.K, a.act,
                             a.accumulate, ctx->dev_error, a3d, b3d, sch));
  FB_LAUNCH_CHECK();
  return FB_OK;
}

template <int BN, int PASSES, bool PAIR, int SG, bool SPLIT>
int32_t launch_layout_sg(fb_ctx* ctx, cudaStream_t stream, const fb_gemm_args& a, const Plan& plan) {
  if (a.a_mn_major) {
    if (a.b_mn_major) return launch_variant<true, true, BN, PASSES, PAIR, SG, SPLIT>(ctx, stream, a, plan);
    return launch_variant<true, false, BN, PASSES, PAIR, SG, SPLIT>(ctx, stream, a, plan);
  }
  if (a.b_mn_major) return launch_variant<false, true, BN, PASSES, PAIR, SG, SPLIT>(ctx, stream, a, plan);
  return launch_variant<false, false, BN, PASSES, PAIR, SG, SPLIT>(ctx, stream, a, plan);
}

// Split-warp groups: the one-CTA tile is bound by shared-memory bandwidth and gains nothing beyond two groups; the
// two-CTA tile is bound by the latency of one split (wait, load, store, proxy fence, remote arrive) and keeps
// gaining up to four (measured 157 -> 175 -> 182 TFLOP/s for 2 -> 3 -> 4 groups at 4096^3).
template <int BN, bool PAIR>
int32_t launch_layout(fb_ctx* ctx, cudaStream_t stream, const fb_gemm_args& a, const Plan& plan) {
  constexpr int SG = PAIR ? 4 : 2;
  return plan.split ? launch_layout_sg<BN, 3, PAIR, SG, true>(ctx, stream, a, plan) : launch_layout_sg<BN, 3, PAIR, SG, false>(ctx, stream, a, plan);
}

// Measured on B200 (4096^3, 3xTF32, persistent kernels): one-CTA 128 x 256 tiles 200-213 TFLOP/s (every MMA re-reads
// all 256 B columns from shared memory), two-CTA 256 x 256 tiles 215-232 TFLOP/s (each CTA reads only its 128 B
// columns).  At 1024 x 4096 x 4096 (one wave of 64 two-CTA tiles on 74 SM pairs) both, and cutting every tile along
// K over all pairs, take 0.204-0.207 ms: what is left there is the unoverlapped prologue and epilogue of a single tile.
//
// How a 3xTF32 product is cut.  Shapes: 128 x 128 (0) and 128 x 256 (1) tiles of one CTA, 256 x 256 tiles of a CTA pair
// (2); ksplit CTAs of one cluster share a tile's K range where whole tiles would leave SMs idle.  The choice is
// the smallest of the modelled times; its constants (us) are fitted to measurements on B200: a k-block of 16 costs
// 0.53 / 0.62 / 0.62, a tile's prologue and epilogue that the next one does not hide 0.5 / 2.5 / 2.5, a launch 5, the
// cluster's reduction 3.5, an accumulation segment that waits for the next one 2.5.  A split runs in one wave (its clusters
// must all fit) so that a slot of the workspace belongs to one CTA.  1024 x 1024 x 16384: 259 -> 158 us; 784 x 512 x 1024:
// 41 -> 17 us; 231 x 512 x 512: 27 -> 12 us.
//
// tail_time: `rest` tiles cut into units of UNIT_KB k-blocks, dealt out over all slots: the units of the longest range, and
// the sums of a tile's parts, which its last CTA adds up by itself (12 us and 5 for each part).  Without the units' rounding
// 7000 x 280 x 592 looked best as 128 x 128 tiles with 17 of 165 in the tail (57 us; 43 as pairs), 1240 x 4960 x 4896 as
// 128 x 256 tiles (350 us; 325 as pairs).
double tail_time(int64_t rest, int64_t slots, int num_kb, double t_kb, double t_tile) {
  const int64_t nu = (num_kb + UNIT_KB - 1) / UNIT_KB;
  if (nu < 2) return 1e30;
  const int64_t units = (rest * nu + slots - 1) / slots;
  const double kb = (double)(units * UNIT_KB < num_kb ? units * UNIT_KB : num_kb);
  return kb * t_kb + t_tile + 12.0 + 5.0 * (double)(nu / units + 1);
}

Plan plan_3xtf32(fb_ctx* ctx, const fb_gemm_args& a, bool force_pair) {
  const int sms = ctx->sm_count - ctx->reserved_sms;
  const int num_kb = (int)((a.K + BK - 1) / BK);
  static const int bm[3] = {128, 128, 256}, bn[3] = {128, 256, 256};
  static const double t_kb[3] = {0.53, 0.62, 0.62}, t_tile[3] = {0.5, 2.5, 2.5};
  Plan best = {1e30, 0, 1, SEG_KB, false, false};
  for (int sh = 2; sh >= 0; --sh) {
    if (sh == 2 && (a.M < 256 || a.N < 256)) continue;
    if (force_pair && sh != 2 && best.time < 1e30) continue;
    if (sh == 1 && a.N <= 128) continue;
    const int ranks = sh == 2 ? 2 : 1;
    const int64_t tiles = ((a.M + bm[sh] - 1) / bm[sh]) * ((a.N + bn[sh] - 1) / bn[sh]);
    for (int lg = 0; lg < 4; ++lg) {
      const int s = 1 << lg;
      double t;
      bool tail = false;
      int seg = SEG_KB, drains = 0;   // of a launch of one wave: accumulation segment, segments before the last
      if (s == 1) {
        const int64_t slots = sms / ranks > 0 ? sms / ranks : 1;
        const int64_t full = tiles / slots, rest = tiles % slots;
        t = 5.0 + full * (num_kb * t_kb[sh] + t_tile[sh]);
        const double whole = num_kb * t_kb[sh] + t_tile[sh];
        if (full == 0) {
          // one wave: whole tiles, or their units over all CTAs
          seg = segment_kblocks(a, num_kb, num_kb, sms, &drains);
          const double cut = tail_time(rest, slots, num_kb, t_kb[sh], t_tile[sh]);
          tail = cut < whole + 2.5 * drains;
          if (tail) { seg = SEG_KB; drains = 0; }
          t += tail ? cut : whole;
        } else if (rest != 0) {
          // A last wave that fills less than 3/4 of the machine is always cut.  (Fuller waves gain nothing: the kernel runs at
          // the power limit, where idle SMs let the busy ones clock higher.)
          tail = 4 * rest < 3 * slots && num_kb > UNIT_KB;
          t += tail ? tail_time(rest, slots, num_kb, t_kb[sh], t_tile[sh]) : whole;
        }
      } else {
        if (sh == 2 || ctx->reserved_sms != 0 || num_kb < 2 * s || tiles > ctx->clusters[lg]) break;
        const int part_kb = (num_kb + s - 1) / s;
        t = 8.5 + part_kb * t_kb[sh] + t_tile[sh];
        seg = segment_kblocks(a, num_kb, part_kb, sms, &drains);
      }
      t += 2.5 * drains;
      if (t < best.time) best = {t, sh, s, seg, s > 1 || drains > 0, tail};
    }
  }
  return best;
}

}  // namespace

bool fb_gemm_tc_supported(const fb_gemm_args& a) {
  if (a.M < 1 || a.N < 1 || a.K < 1) return false;
  if (a.M > 0x7fffff00 || a.N > 0x7fffff00 || a.K > 0x7fffff00) return false;
  if (a.bias_m != nullptr) return false;
  if (!fb_aligned16(a.A) || !fb_aligned16(a.B) || !fb_aligned16(a.C)) return false;
  if (a.Z && !fb_aligned16(a.Z)) return false;
  if (a.bias_n && !fb_aligned16(a.bias_n)) return false;
  if (a.lda % 4 || a.ldb % 4 || a.ldc % 4) return false;
  // the leading dimension must cover the contiguous extent
  if (a.lda < (a.a_mn_major ? a.M : a.K) || a.ldb < (a.b_mn_major ? a.N : a.K) || a.ldc < a.N) return false;
  return true;
}

double fb_gemm_tc_time(fb_ctx* ctx, const fb_gemm_args& a) { return plan_3xtf32(ctx, a, false).time; }

// passes: 3 = 3xTF32, 1 = one TF32 pass, 32 = 3xTF32 on two-CTA tiles where the shape allows
int32_t fb_gemm_tc_launch(fb_ctx* ctx, cudaStream_t stream, const fb_gemm_args& a, int passes, const int32_t* run_if) {
  if (!fb_gemm_tc_supported(a)) return FB_ERR_UNSUPPORTED;
  if (passes == 1) {
    const bool narrow1 = (a.N <= 128) || (2 * ((a.M + BM - 1) / BM) * ((a.N + 255) / 256) <= ctx->sm_count);
    // (TF32 in one pass: the last wave is cut as it always was)
    const int64_t slots = ctx->sm_count - ctx->reserved_sms, rest = (((a.M + BM - 1) / BM) * ((a.N + (narrow1 ? 127 : 255)) / (narrow1 ? 128 : 256))) % slots;
    const Plan whole = {0.0, 0, 1, SEG_KB, false, rest != 0 && 4 * rest < 3 * slots && a.K > BK * UNIT_KB, run_if};
    return narrow1 ? launch_layout_sg<128, 1, false, 2, false>(ctx, stream, a, whole) : launch_layout_sg<256, 1, false, 2, false>(ctx, stream, a, whole);
  }
  Plan p = plan_3xtf32(ctx, a, passes == 32);
  p.run_if = run_if;
  if (p.shape == 0) return launch_layout<128, false>(ctx, stream, a, p);
  if (p.shape == 1) return launch_layout<256, false>(ctx, stream, a, p);
  return launch_layout<256, true>(ctx, stream, a, p);
}

// How many clusters of 2, 4 and 8 CTAs with the GEMM's shared memory are resident at once (called by fb_ctx_create).
void fb_gemm_query_clusters(fb_ctx* ctx) {
  auto kern = gemm_tc_kernel<false, true, 256, 3, false, 2, true>;
  using cfg = Cfg<256, 3, false, 2>;
  ctx->clusters[0] = ctx->sm_count;
  for (int lg = 1; lg < 4; ++lg) {
    ctx->clusters[lg] = 0;
    cudaLaunchConfig_t lc;
    memset(&lc, 0, sizeof(lc));
    lc.gridDim = dim3((unsigned)(ctx->sm_count / (1 << lg) * (1 << lg)), 1, 1);
    lc.blockDim = dim3(cfg::NUM_THREADS, 1, 1);
    lc.dynamicSmemBytes = cfg::SMEM_BYTES;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 1u << lg;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    lc.attrs = attr;
    lc.numAttrs = 1;
    int n = 0;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, cfg::SMEM_BYTES) == cudaSuccess &&
        cudaOccupancyMaxActiveClusters(&n, kern, &lc) == cudaSuccess)
      ctx->clusters[lg] = n;
    else
      cudaGetLastError();
  }
}
