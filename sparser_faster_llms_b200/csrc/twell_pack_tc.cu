// Gate projection + ReLU + TwELL pack on the 5th-generation tensor cores.
//
// Kernels of this file: twell_pack_tc_splitk_(wide_)kernel (17..32 tokens) and, only where a caller asks for it,
// twell_pack_tc_splitk_mid_kernel (128-token tiles), both with D split over a cluster.
// Larger calls run on one-SM tiles (tile_mlp.cu) and on pairs of SMs (pair_gemm.cuh).
//
// CTA tile: one 256-neuron TwELL tile x NTOK tokens x a slice of D.
// Neurons ride the MMA M axis as two 128-row accumulators, tokens the N axis:
//   D0[128, NTOK] = W[tile*256      .. +128, :] . X[tok0 .. +NTOK, :]^T
//   D1[128, NTOK] = W[tile*256 + 128 .. +128, :] . X[tok0 .. +NTOK, :]^T
// Operands are K-major bf16 tiles of 64 k-values (128 bytes per row), brought in by
// TMA (cp.async.bulk.tensor, 128-byte swizzle, no multicast) into a ring of shared
// memory stages; one elected thread issues tcgen05.mma (kind::f16, fp32 accumulate
// in TMEM); tcgen05.commit releases a stage back to the producer and, after the
// last k step, hands the accumulators to the epilogue warps.
//
// In TMEM a lane is a neuron and a column is a token, so after tcgen05.ld the 32
// lanes of an epilogue warp hold 32 consecutive neurons of one token per register:
// __ballot_sync gives the tile's positives in ascending neuron order, __popc the
// slot.  Eight (accumulator, warp) chunks per token are stitched by an exclusive
// prefix in shared memory.  Deterministic; same slab bytes as the small-M kernel.
//
// Every mbarrier wait is bounded: when a wait gives up, the CTA raises an error word
// (read with b200_twell_pack_tc_status), skips the rest of its work, frees its TMEM
// and returns.
//
// Replaces mm_wgmma_nt_kernel (custom_models/twell_modules/matmul_d2t.cu:287-709):
// wgmma -> tcgen05.mma, register accumulators -> TMEM, multicast TMA -> per-CTA TMA,
// shared-memory atomics in the epilogue -> ballot/popc.
#include <cooperative_groups.h>

#include <cstdlib>

#include "tc_common.cuh"

namespace cg = cooperative_groups;

namespace b200 {

int pair_gemm_status();
int tile_mlp_status();

namespace {

__device__ int g_tc_error = 0;

// ---------------------------------------------------------------------------
// Decode variant (M <= 32): the TMA -> tcgen05 pipeline with the reduction
// dimension split over a cluster of CL CTAs so that (H/256)*CL CTAs stream W_gate
// concurrently.  CTA `crank` multiplies all 256 neurons of the tile by its slice of D for
// up to 32 tokens; the partial accumulators leave TMEM through registers and are pushed
// (distributed shared memory) to the CTA that finalises each token, which adds the CL
// partials in rank order and compacts with ballot / popc.
// grid = ((H/256) * CL, ceil(M / 32)), cluster = CL.
// Dynamic shared memory: STAGES x (A0 | A1 | B) | partial sums [32][kPartStrideTc] fp32.
// ---------------------------------------------------------------------------
constexpr int kTokDecode = 32;
constexpr int kPartStrideTc = kTileN + 4;

template <int CL, int STAGES>
__global__ void __launch_bounds__(kThreadsTc, CL >= 8 ? 2 : 1)
twell_pack_tc_splitk_kernel(const __grid_constant__ CUtensorMap tmap_w,
                            const __grid_constant__ CUtensorMap tmap_x,
                            const float* __restrict__ bias, uint32_t* __restrict__ packed, int M,
                            int D, int slab_w, int row_words) {
  constexpr int NTOK = kTokDecode;
  constexpr int TOK = NTOK / CL;  // tokens finalised by this CTA
  constexpr int kBTileBytes = NTOK * 128;
  constexpr int kStageBytes = 2 * kATileBytes + kBTileBytes;
  constexpr uint32_t kTmemCols = 2 * NTOK;
  constexpr uint32_t kIdesc = umma_idesc(128, NTOK);
  constexpr int EPT = TOK * kTileN / 128;  // elements per epilogue thread in the final pass

  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  float* part = reinterpret_cast<float*>(smem + (size_t)STAGES * kStageBytes);
  __shared__ __align__(8) uint64_t full_bar[STAGES], empty_bar[STAGES], acc_bar;
  __shared__ uint32_t tmem_slot;
  __shared__ volatile int abort_s;
  __shared__ int cnt_chunk[TOK][8];

  cg::cluster_group cluster = cg::this_cluster();
  const int crank = (int)cluster.block_rank();
  cluster.barrier_arrive();  // matched by barrier_wait() before the first remote store

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int tile = blockIdx.x / CL;
  const int m0 = blockIdx.y * NTOK;
  const int kc = D / CL;
  const int ksteps = kc / kStageK;
  const int k_base = crank * kc;

  if (threadIdx.x == 0) {
#pragma unroll
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    mbar_init(&acc_bar, 1);
    abort_s = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                 ::"r"(smem_u32(&tmem_slot)), "r"(kTmemCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_base = tmem_slot;
  // Barriers, TMEM and the cluster hand-shake are set up; from here on the kernel reads x and
  // writes the slab, so the predecessor in the stream must have completed.
  pdl_wait();

  if (warp == 0) {
    if (elect_one() &&
        !ring_produce<STAGES>(full_bar, empty_bar, ksteps, kStageBytes, [&](int k, int s) {
          unsigned char* st = smem + (size_t)s * kStageBytes;
          const int kcoord = k_base + k * kStageK;
          // one copy for the tile's 256 weight rows (A0 | A1 are contiguous)
          tma_load_2d(st, &tmap_w, kcoord, tile * kTileN, &full_bar[s]);
          tma_load_2d(st + 2 * kATileBytes, &tmap_x, kcoord, m0, &full_bar[s]);
        })) {
      abort_s = 1;
      atomicExch(&g_tc_error, 1);
    }
  } else if (warp == 1) {
    const uint64_t d0 = umma_desc(smem_u32(smem));
    if (elect_one()) {
      const bool done = ring_issue<STAGES>(full_bar, empty_bar, ksteps, [&](bool first, int s) {
        const uint64_t da0 = d0 + (uint32_t)s * (kStageBytes >> 4), da1 = da0 + (kATileBytes >> 4),
                       db = da0 + (2 * kATileBytes >> 4);
#pragma unroll
        for (int kk = 0; kk < kStageK / 16; ++kk) {
          const uint32_t acc = !first || kk > 0 ? 1u : 0u;
          umma_bf16(tmem_base, da0 + 2 * kk, db + 2 * kk, kIdesc, acc);
          umma_bf16(tmem_base + NTOK, da1 + 2 * kk, db + 2 * kk, kIdesc, acc);
        }
      });
      if (done) {
        umma_commit(&acc_bar);
      } else {
        abort_s = 1;
        atomicExch(&g_tc_error, 2);
      }
    }
  } else {
    // ---- epilogue part 1: TMEM -> registers -> owner CTA's shared memory ----
    const int q = warp & 3;
    bool ok = mbar_wait(&acc_bar, 0u);
    if (!ok) {
      abort_s = 1;
      atomicExch(&g_tc_error, 3);
    }
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    cluster.barrier_wait();  // every CTA of the cluster is running
    if (ok) {
      const int nl = q * 32 + lane;  // neuron inside the tile (accumulator 0); +128 for 1
      const uint32_t lane_addr = tmem_base + ((uint32_t)(q * 32) << 16);
      float v0[32], v1[32];
      tmem_ld32(lane_addr, v0);
      tmem_ld32(lane_addr + (uint32_t)NTOK, v1);
#pragma unroll
      for (int c = 0; c < NTOK; ++c) {
        const int owner = c / TOK, tl = c % TOK;
        float* dst = cluster.map_shared_rank(part, owner) +
                     (size_t)(crank * TOK + tl) * kPartStrideTc + nl;
        dst[0] = v0[c];
        dst[128] = v1[c];
      }
    }
  }
  if (warp < 2) cluster.barrier_wait();  // pair the early arrive for the non-epilogue warps

  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  cluster.sync();  // all partials delivered (every thread of every CTA takes part)
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base),
                 "r"(kTmemCols)
                 : "memory");
  }
  if (warp < 2 || abort_s) return;

  // ---- epilogue part 2: this CTA finalises tokens [crank*TOK, (crank+1)*TOK) ----
  const int et = threadIdx.x - 64;
  const int neuron0 = tile * kTileN;
  float z[EPT];
  uint32_t mask[EPT];
#pragma unroll
  for (int i = 0; i < EPT; ++i) {
    const int e = et + i * 128;
    const int tl = e / kTileN, nl = e % kTileN;
    const int tok = crank * TOK + tl;
    float v = 0.f;
#pragma unroll
    for (int r = 0; r < CL; ++r) v += part[(size_t)(r * TOK + tl) * kPartStrideTc + nl];
    if (bias != nullptr) v += bias[neuron0 + nl];
    const bool keep = (v > 0.f) && (m0 + tok < M);
    z[i] = v;
    mask[i] = __ballot_sync(0xffffffffu, keep);
    if (lane == 0) cnt_chunk[tl][nl / 32] = __popc(mask[i]);
  }
  epi_barrier();
  if (et < TOK) {  // counts -> exclusive prefix over the 8 chunks of this token, count word
    int run = 0;
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      const int v = cnt_chunk[et][c];
      cnt_chunk[et][c] = run;
      run += v;
    }
    const int tok = m0 + crank * TOK + et;
    if (tok < M) packed[(size_t)tok * row_words + (size_t)tile * slab_w] = (uint32_t)run;
  }
  epi_barrier();
#pragma unroll
  for (int i = 0; i < EPT; ++i) {
    const int e = et + i * 128;
    const int tl = e / kTileN, nl = e % kTileN;
    const int tok = crank * TOK + tl;
    if (m0 + tok >= M) continue;
    uint32_t* slab = packed + (size_t)(m0 + tok) * row_words + (size_t)tile * slab_w;
    const int slot = cnt_chunk[tl][nl / 32] + __popc(mask[i] & lanemask_lt());
    if (((mask[i] >> lane) & 1u) && slot < slab_w - 1)
      slab[1 + slot] = (uint32_t)(neuron0 + nl) | (bf16_bits(z[i]) << 16);
  }
}

// ---------------------------------------------------------------------------
// The same split-k kernel with sixteen epilogue warps instead of four.  The epilogue of the
// four-warp form is a latency chain on one warp per scheduler (TMEM read, 64 remote stores
// per thread, then 16 elements per thread to sum, ballot and store).  Here four groups of
// four warps each read 8 token columns of their TMEM lane quarter (tcgen05.ld ...x8) and push
// 16 values per thread, and all 512 epilogue threads take part in the final pass (4 elements
// per thread for a 4-CTA cluster).  Same arithmetic, same slab bytes.
// Threads: warp 0 producer, warp 1 mma, warps 2..17 epilogue (group = (warp - 2) / 4, TMEM
// lane quarter = warp % 4).
// ---------------------------------------------------------------------------
constexpr int kThreadsTcWide = 64 + 512;

template <int CL, int STAGES>
__global__ void __launch_bounds__(kThreadsTcWide, 1)
twell_pack_tc_splitk_wide_kernel(const __grid_constant__ CUtensorMap tmap_w,
                                 const __grid_constant__ CUtensorMap tmap_x,
                                 const float* __restrict__ bias, uint32_t* __restrict__ packed,
                                 int M, int D, int slab_w, int row_words) {
  constexpr int NTOK = kTokDecode;
  constexpr int TOK = NTOK / CL;
  constexpr int kBTileBytes = NTOK * 128;
  constexpr int kStageBytes = 2 * kATileBytes + kBTileBytes;
  constexpr uint32_t kTmemCols = 2 * NTOK;
  constexpr uint32_t kIdesc = umma_idesc(128, NTOK);
  constexpr int EPT = TOK * kTileN / 512;  // elements per epilogue thread in the final pass
  static_assert(EPT >= 1, "the final pass needs at least one element per thread");

  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  float* part = reinterpret_cast<float*>(smem + (size_t)STAGES * kStageBytes);
  __shared__ __align__(8) uint64_t full_bar[STAGES], empty_bar[STAGES], acc_bar;
  __shared__ uint32_t tmem_slot;
  __shared__ volatile int abort_s;
  __shared__ int cnt_chunk[TOK][8];

  cg::cluster_group cluster = cg::this_cluster();
  const int crank = (int)cluster.block_rank();
  cluster.barrier_arrive();  // matched by barrier_wait() before the first remote store

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int tile = blockIdx.x / CL;
  const int m0 = blockIdx.y * NTOK;
  const int kc = D / CL;
  const int ksteps = kc / kStageK;
  const int k_base = crank * kc;

  if (threadIdx.x == 0) {
#pragma unroll
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    mbar_init(&acc_bar, 1);
    abort_s = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                 ::"r"(smem_u32(&tmem_slot)), "r"(kTmemCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_base = tmem_slot;
  if (threadIdx.x == 0)  // two of the eight k-steps at D 2048: one is slower (724 us), three level
    for (int k = 0; k < 2 && k < ksteps; ++k)
      tma_prefetch_2d(&tmap_w, k_base + k * kStageK, tile * kTileN);
  pdl_wait();

  if (warp == 0) {
    if (elect_one() &&
        !ring_produce<STAGES>(full_bar, empty_bar, ksteps, kStageBytes, [&](int k, int s) {
          unsigned char* st = smem + (size_t)s * kStageBytes;
          const int kcoord = k_base + k * kStageK;
          // one copy for the tile's 256 weight rows (A0 | A1 are contiguous)
          tma_load_2d(st, &tmap_w, kcoord, tile * kTileN, &full_bar[s]);
          tma_load_2d(st + 2 * kATileBytes, &tmap_x, kcoord, m0, &full_bar[s]);
        })) {
      abort_s = 1;
      atomicExch(&g_tc_error, 1);
    }
  } else if (warp == 1) {
    const uint64_t d0 = umma_desc(smem_u32(smem));
    if (elect_one()) {
      const bool done = ring_issue<STAGES>(full_bar, empty_bar, ksteps, [&](bool first, int s) {
        const uint64_t da0 = d0 + (uint32_t)s * (kStageBytes >> 4), da1 = da0 + (kATileBytes >> 4),
                       db = da0 + (2 * kATileBytes >> 4);
#pragma unroll
        for (int kk = 0; kk < kStageK / 16; ++kk) {
          const uint32_t acc = !first || kk > 0 ? 1u : 0u;
          umma_bf16(tmem_base, da0 + 2 * kk, db + 2 * kk, kIdesc, acc);
          umma_bf16(tmem_base + NTOK, da1 + 2 * kk, db + 2 * kk, kIdesc, acc);
        }
      });
      if (done) {
        umma_commit(&acc_bar);
      } else {
        abort_s = 1;
        atomicExch(&g_tc_error, 2);
      }
    }
  } else {
    // ---- epilogue part 1: TMEM -> registers -> owner CTA's shared memory ----
    const int q = warp & 3;
    const int grp = (warp - 2) >> 2;  // token columns [8 * grp, 8 * grp + 8)
    bool ok = mbar_wait(&acc_bar, 0u);
    if (!ok) {
      abort_s = 1;
      atomicExch(&g_tc_error, 3);
    }
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    cluster.barrier_wait();  // every CTA of the cluster is running
    if (ok) {
      const int nl = q * 32 + lane;  // neuron inside the tile (accumulator 0); +128 for 1
      const uint32_t lane_addr = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(grp * 8);
      float v0[8], v1[8];
      tmem_ld8(lane_addr, v0);
      tmem_ld8(lane_addr + (uint32_t)NTOK, v1);
#pragma unroll
      for (int c8 = 0; c8 < 8; ++c8) {
        const int c = grp * 8 + c8;
        const int owner = c / TOK, tl = c % TOK;
        float* dst = cluster.map_shared_rank(part, owner) +
                     (size_t)(crank * TOK + tl) * kPartStrideTc + nl;
        dst[0] = v0[c8];
        dst[128] = v1[c8];
      }
    }
  }
  if (warp < 2) cluster.barrier_wait();  // pair the early arrive for the non-epilogue warps

  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  cluster.sync();  // all partials delivered (every thread of every CTA takes part)
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base),
                 "r"(kTmemCols)
                 : "memory");
  }
  if (warp < 2 || abort_s) return;

  // ---- epilogue part 2: this CTA finalises tokens [crank*TOK, (crank+1)*TOK) ----
  const int et = threadIdx.x - 64;  // 0..511
  const int neuron0 = tile * kTileN;
  float z[EPT];
  uint32_t mask[EPT];
#pragma unroll
  for (int i = 0; i < EPT; ++i) {
    const int e = et + i * 512;
    const int tl = e / kTileN, nl = e % kTileN;
    const int tok = crank * TOK + tl;
    float v = 0.f;
#pragma unroll
    for (int r = 0; r < CL; ++r) v += part[(size_t)(r * TOK + tl) * kPartStrideTc + nl];
    if (bias != nullptr) v += bias[neuron0 + nl];
    const bool keep = (v > 0.f) && (m0 + tok < M);
    z[i] = v;
    mask[i] = __ballot_sync(0xffffffffu, keep);
    if (lane == 0) cnt_chunk[tl][nl / 32] = __popc(mask[i]);
  }
  named_barrier2(512);
  if (et < TOK) {  // counts -> exclusive prefix over the 8 chunks of this token, count word
    int run = 0;
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      const int v = cnt_chunk[et][c];
      cnt_chunk[et][c] = run;
      run += v;
    }
    const int tok = m0 + crank * TOK + et;
    if (tok < M) packed[(size_t)tok * row_words + (size_t)tile * slab_w] = (uint32_t)run;
  }
  named_barrier2(512);
#pragma unroll
  for (int i = 0; i < EPT; ++i) {
    const int e = et + i * 512;
    const int tl = e / kTileN, nl = e % kTileN;
    const int tok = crank * TOK + tl;
    if (m0 + tok >= M) continue;
    uint32_t* slab = packed + (size_t)(m0 + tok) * row_words + (size_t)tile * slab_w;
    const int slot = cnt_chunk[tl][nl / 32] + __popc(mask[i] & lanemask_lt());
    if (((mask[i] >> lane) & 1u) && slot < slab_w - 1)
      slab[1 + slot] = (uint32_t)(neuron0 + nl) | (bf16_bits(z[i]) << 16);
  }
}

// ---------------------------------------------------------------------------
// Split-k kernel for 33..256 tokens: the decode kernel above with 128-token tiles.  A tile of
// 256 neurons x 128 tokens has only H / 256 CTAs to itself when d_model is not split (32 at
// d_ff 8192: 32 SMs walking 32 latency-bound k-steps, 31-36 us per call whatever the token
// count); split four ways over a cluster every SM streams a quarter of the weight rows.
// The fp32 partial tile of a CTA (128 KB) does not fit next to the operand ring, so the
// partial sums land in the ring itself: a cluster barrier after every CTA's last MMA (instead
// of the early arrive of the decode kernel) makes the ring free, then the TMEM -> DSMEM push,
// a second cluster barrier and the same final pass (CTA r owns 128 / CL tokens).
// grid = ((H/256) * CL, ceil(M / 128)), cluster = CL (4, or 2 when four CTAs per tile would not
// fit one wave), 576 threads.
// ---------------------------------------------------------------------------
constexpr int kTokMid = 128;

template <int CL, int STAGES>
__global__ void __launch_bounds__(kThreadsTcWide, 1)
twell_pack_tc_splitk_mid_kernel(const __grid_constant__ CUtensorMap tmap_w,
                                const __grid_constant__ CUtensorMap tmap_x,
                                const float* __restrict__ bias, uint32_t* __restrict__ packed,
                                int M, int D, int slab_w, int row_words) {
  constexpr int NTOK = kTokMid;
  constexpr int TOK = NTOK / CL;  // tokens finalised per CTA: 32 (CL 4) or 64 (CL 2)
  static_assert(CL == 2 || CL == 4, "cluster size");
  constexpr int kBTileBytes = NTOK * 128;
  constexpr int kStageBytes = 2 * kATileBytes + kBTileBytes;
  constexpr uint32_t kTmemCols = 2 * NTOK;
  constexpr uint32_t kIdesc = umma_idesc(128, NTOK);
  constexpr int EPT = TOK * kTileN / 512;  // elements per epilogue thread in the final pass
  static_assert((size_t)NTOK * kPartStrideTc * sizeof(float) <= (size_t)STAGES * kStageBytes,
                "the partial sums must fit into the operand ring");

  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  float* part = reinterpret_cast<float*>(smem);  // [CL source ranks x TOK][kPartStrideTc], after the ring is free
  __shared__ __align__(8) uint64_t full_bar[STAGES], empty_bar[STAGES], acc_bar;
  __shared__ uint32_t tmem_slot;
  __shared__ volatile int abort_s;
  __shared__ int cnt_chunk[TOK][8];

  cg::cluster_group cluster = cg::this_cluster();
  const int crank = (int)cluster.block_rank();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int tile = blockIdx.x / CL;
  const int m0 = blockIdx.y * NTOK;
  const int kc = D / CL;
  const int ksteps = kc / kStageK;
  const int k_base = crank * kc;

  if (threadIdx.x == 0) {
#pragma unroll
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    mbar_init(&acc_bar, 1);
    abort_s = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                 ::"r"(smem_u32(&tmem_slot)), "r"(kTmemCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_base = tmem_slot;
  if (threadIdx.x == 0)  // 37 tokens, H 5632, eager layers: 26.8 -> 26.4 us; 128, H 8192: 48.0 -> 47.4
    for (int k = 0; k < 2 && k < ksteps; ++k)
      tma_prefetch_2d(&tmap_w, k_base + k * kStageK, tile * kTileN);
  pdl_wait();

  bool ok = true;
  if (warp == 0) {
    if (elect_one() &&
        !ring_produce<STAGES>(full_bar, empty_bar, ksteps, kStageBytes, [&](int k, int s) {
          unsigned char* st = smem + (size_t)s * kStageBytes;
          const int kcoord = k_base + k * kStageK;
          tma_load_2d(st, &tmap_w, kcoord, tile * kTileN, &full_bar[s]);  // 256 rows: A0 | A1
          tma_load_2d(st + 2 * kATileBytes, &tmap_x, kcoord, m0, &full_bar[s]);
        })) {
      abort_s = 1;
      atomicExch(&g_tc_error, 1);
    }
  } else if (warp == 1) {
    const uint64_t d0 = umma_desc(smem_u32(smem));
    if (elect_one()) {
      const bool done = ring_issue<STAGES>(full_bar, empty_bar, ksteps, [&](bool first, int s) {
        const uint64_t da0 = d0 + (uint32_t)s * (kStageBytes >> 4), da1 = da0 + (kATileBytes >> 4),
                       db = da0 + (2 * kATileBytes >> 4);
#pragma unroll
        for (int kk = 0; kk < kStageK / 16; ++kk) {
          const uint32_t acc = !first || kk > 0 ? 1u : 0u;
          umma_bf16(tmem_base, da0 + 2 * kk, db + 2 * kk, kIdesc, acc);
          umma_bf16(tmem_base + NTOK, da1 + 2 * kk, db + 2 * kk, kIdesc, acc);
        }
      });
      if (done) {
        umma_commit(&acc_bar);
      } else {
        abort_s = 1;
        atomicExch(&g_tc_error, 2);
      }
    }
  } else {
    // every MMA of this CTA has read its operands once the accumulators are published
    ok = mbar_wait(&acc_bar, 0u);
    if (!ok) {
      abort_s = 1;
      atomicExch(&g_tc_error, 3);
    }
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  }
  // Every CTA of the cluster is past its last MMA (or has given up): the rings are free.
  cluster.sync();

  if (warp >= 2 && ok) {
    // ---- epilogue part 1: TMEM -> registers -> the owner's ring memory ----
    const int q = warp & 3;
    const int grp = (warp - 2) >> 2;  // token columns [32 grp, 32 grp + 32)
    const int owner = grp * 32 / TOK, tl0 = grp * 32 % TOK;
    const int nl = q * 32 + lane;     // neuron inside the tile (accumulator 0); +128 for 1
    const uint32_t lane_addr = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(grp * 32);
    float* dst0 = cluster.map_shared_rank(part, owner) +
                  (size_t)(crank * TOK + tl0) * kPartStrideTc + nl;
    float v[32];
    tmem_ld32(lane_addr, v);
#pragma unroll
    for (int c = 0; c < 32; ++c) dst0[(size_t)c * kPartStrideTc] = v[c];
    tmem_ld32(lane_addr + (uint32_t)NTOK, v);
#pragma unroll
    for (int c = 0; c < 32; ++c) dst0[(size_t)c * kPartStrideTc + 128] = v[c];
  }

  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  cluster.sync();  // all partials delivered (every thread of every CTA takes part)
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base),
                 "r"(kTmemCols)
                 : "memory");
  }
  if (warp < 2 || abort_s) return;

  // ---- epilogue part 2: this CTA finalises tokens [crank*TOK, (crank+1)*TOK) ----
  const int et = threadIdx.x - 64;  // 0..511
  const int neuron0 = tile * kTileN;
  float z[EPT];
  uint32_t mask[EPT];
#pragma unroll
  for (int i = 0; i < EPT; ++i) {
    const int e = et + i * 512;
    const int tl = e / kTileN, nl = e % kTileN;
    const int tok = crank * TOK + tl;
    float v = 0.f;
#pragma unroll
    for (int r = 0; r < CL; ++r) v += part[(size_t)(r * TOK + tl) * kPartStrideTc + nl];
    if (bias != nullptr) v += bias[neuron0 + nl];
    const bool keep = (v > 0.f) && (m0 + tok < M);
    z[i] = v;
    mask[i] = __ballot_sync(0xffffffffu, keep);
    if (lane == 0) cnt_chunk[tl][nl / 32] = __popc(mask[i]);
  }
  named_barrier2(512);
  if (et < TOK) {  // counts -> exclusive prefix over the 8 chunks of this token, count word
    int run = 0;
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      const int v = cnt_chunk[et][c];
      cnt_chunk[et][c] = run;
      run += v;
    }
    const int tok = m0 + crank * TOK + et;
    if (tok < M) packed[(size_t)tok * row_words + (size_t)tile * slab_w] = (uint32_t)run;
  }
  named_barrier2(512);
#pragma unroll
  for (int i = 0; i < EPT; ++i) {
    const int e = et + i * 512;
    const int tl = e / kTileN, nl = e % kTileN;
    const int tok = crank * TOK + tl;
    if (m0 + tok >= M) continue;
    uint32_t* slab = packed + (size_t)(m0 + tok) * row_words + (size_t)tile * slab_w;
    const int slot = cnt_chunk[tl][nl / 32] + __popc(mask[i] & lanemask_lt());
    if (((mask[i] >> lane) & 1u) && slot < slab_w - 1)
      slab[1 + slot] = (uint32_t)(neuron0 + nl) | (bf16_bits(z[i]) << 16);
  }
}

// ---- host side -------------------------------------------------------------
template <int CL, int STAGES>
int launch_tc_splitk_mid(const void* x, const void* w, const float* bias, void* packed, int64_t M,
                         int64_t D, int64_t H, int cf, cudaStream_t stream) {
  CUtensorMap map_w, map_x;
  if (int rc = make_map(&map_w, w, H, D, 256)) return rc;
  if (int rc = make_map(&map_x, x, M, D, kTokMid)) return rc;
  const size_t smem = (size_t)STAGES * (2 * kATileBytes + kTokMid * 128) + 1024;
  auto kern = twell_pack_tc_splitk_mid_kernel<CL, STAGES>;
  static size_t granted[64] = {0};
  if (int rc = ensure_dynamic_smem(kern, smem, granted, "b200_twell_pack")) return rc;
  const int slab_w = kTileN / cf;
  const int tiles = (int)(H / kTileN);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(tiles * CL), (unsigned)((M + kTokMid - 1) / kTokMid), 1);
  cfg.blockDim = dim3(kThreadsTcWide, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = CL;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = add_pdl_attribute(attr, 1, 1);
  cudaError_t e = cudaLaunchKernelEx(&cfg, kern, map_w, map_x, bias,
                                     static_cast<uint32_t*>(packed), (int)M, (int)D, slab_w,
                                     tiles * slab_w);
  if (e != cudaSuccess)
    return fail(B200_ECUDA, "b200_twell_pack (tcgen05 split-k, 128-token tiles): launch: %s",
                cudaGetErrorString(e));
  return B200_OK;
}

// Epilogue form of the split-k kernel: sixteen epilogue warps unless B200_PACK_WIDE=0.
bool pack_wide_enabled() {
  static int on = -1;
  if (on < 0) {
    const char* e = getenv("B200_PACK_WIDE");
    on = (e != nullptr && atoi(e) == 0) ? 0 : 1;
  }
  return on != 0;
}

template <int CL, int STAGES, bool WIDE>
int launch_tc_splitk_form(const void* x, const void* w, const float* bias, void* packed,
                          int64_t M, int64_t D, int64_t H, int cf, cudaStream_t stream) {
  CUtensorMap map_w, map_x;
  if (int rc = make_map(&map_w, w, H, D, 256)) return rc;
  if (int rc = make_map(&map_x, x, M, D, kTokDecode)) return rc;
  const size_t smem = (size_t)STAGES * (2 * kATileBytes + kTokDecode * 128) +
                      (size_t)kTokDecode * kPartStrideTc * sizeof(float) + 1024;
  auto kern = WIDE ? twell_pack_tc_splitk_wide_kernel<CL, STAGES>
                   : twell_pack_tc_splitk_kernel<CL, STAGES>;
  static size_t granted[64] = {0};
  if (int rc = ensure_dynamic_smem(kern, smem, granted, "b200_twell_pack")) return rc;
  const int slab_w = kTileN / cf;
  const int tiles = (int)(H / kTileN);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(tiles * CL), (unsigned)((M + kTokDecode - 1) / kTokDecode), 1);
  cfg.blockDim = dim3(WIDE ? kThreadsTcWide : kThreadsTc, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = CL;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = add_pdl_attribute(attr, 1, 1);
  cudaError_t e = cudaLaunchKernelEx(&cfg, kern, map_w, map_x, bias,
                                     static_cast<uint32_t*>(packed), (int)M, (int)D, slab_w,
                                     tiles * slab_w);
  if (e != cudaSuccess)
    return fail(B200_ECUDA, "b200_twell_pack (tcgen05 split-k): launch: %s",
                cudaGetErrorString(e));
  return B200_OK;
}

template <int CL, int STAGES>
int launch_tc_splitk(const void* x, const void* w, const float* bias, void* packed, int64_t M,
                     int64_t D, int64_t H, int cf, cudaStream_t stream) {
  return pack_wide_enabled()
             ? launch_tc_splitk_form<CL, STAGES, true>(x, w, bias, packed, M, D, H, cf, stream)
             : launch_tc_splitk_form<CL, STAGES, false>(x, w, bias, packed, M, D, H, cf, stream);
}

}  // namespace

// Decode path on the tensor cores: split-k over a cluster of 4 CTAs.
int twell_pack_tc_splitk(const void* x, const void* w, const float* bias, void* packed, int64_t M,
                         int64_t D, int64_t H, int cf, cudaStream_t stream) {
  return launch_tc_splitk<4, 5>(x, w, bias, packed, M, D, H, cf, stream);
}

// The same with D split 8 ways: twice the CTAs for narrow d_ff (a d_ff shard of 2048..4096
// neurons has only 8..16 tiles).  Needs D % 512 == 0.
int twell_pack_tc_splitk8(const void* x, const void* w, const float* bias, void* packed,
                          int64_t M, int64_t D, int64_t H, int cf, cudaStream_t stream) {
  if (D % 512) return fail(B200_EUNSUPPORTED, "b200_twell_pack: 8-way split needs D %% 512 == 0");
  return launch_tc_splitk<8, 4>(x, w, bias, packed, M, D, H, cf, stream);
}

// (A 2-way split - 64 CTAs streaming 512 KB each at H = 8192 - was measured at 16.8 us against
// 12.8 us for the 4-way split: one SM pulls about 64 GB/s through TMA, so the weight stream
// needs well over 100 CTAs to reach the HBM rate.)

// 33..256 tokens: split-k over a cluster of `split` (4 or 2) CTAs with 128-token tiles.  Only by choice of the
// caller: the one-SM tiles of tile_mlp.cu are level or ahead at every size.
int twell_pack_tc_splitk_mid(const void* x, const void* w, const float* bias, void* packed,
                             int64_t M, int64_t D, int64_t H, int cf, int split,
                             cudaStream_t stream) {
  if (split == 2) return launch_tc_splitk_mid<2, 4>(x, w, bias, packed, M, D, H, cf, stream);
  return launch_tc_splitk_mid<4, 4>(x, w, bias, packed, M, D, H, cf, stream);
}

// Error word raised by a bounded wait that gave up (0 = none).  Reads and clears it;
// synchronises the device.
int twell_pack_tc_status() {
  int v = 0, zero = 0;
  if (cudaMemcpyFromSymbol(&v, g_tc_error, sizeof(int)) != cudaSuccess) return -1;
  if (v != 0) cudaMemcpyToSymbol(g_tc_error, &zero, sizeof(int));
  const int pair = pair_gemm_status(), tile = tile_mlp_status();
  return v != 0 ? v : pair != 0 ? pair : tile;
}

}  // namespace b200
