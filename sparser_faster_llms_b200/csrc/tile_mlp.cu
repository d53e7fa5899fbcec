// The fused MLPs for some dozens to some hundreds of tokens: two launches of one-SM tensor-core tiles
// that fill the GPU where the 256 x 256 tiles of the paired GEMM (pair_gemm.cuh) would leave most of it
// idle.
//
//   first    CTA = 128 tokens x NB neurons (64 or 128) of the gate and of the up product, both in one
//            accumulator of 2 NB columns; the CTAs of a 256-neuron slab tile form a cluster and
//            exchange their stored counts, so every CTA knows the slots of its entries.  Writes the
//            slabs and hidden = relu(gate) * up on the stored pattern.
//   second   CTA = 128 tokens x ND output columns x a slice of the neurons; a cluster of CL CTAs holds
//            all slices.  Every CTA hands each owner its 128 x ND / CL fp32 sums through distributed
//            shared memory, the owner adds them in rank order and stores.
//
// What bounds both: the weights' stream and, per SM, the 64 bytes a clock that TMA brings into shared
// memory, so the split is the one that puts the weights on as many SMs as fit one wave.  The gather form
// has two latency chains of four to six round trips behind the same stream, and its rows come through
// L2 once per token.
//
// Threads (352): warp 0 loads weights, warp 1 tokens, warp 2 issues the MMAs, warps 3..10 epilogue, two
// per TMEM lane quarter (lane = token).  Every wait is bounded; one that gives up sets the error word,
// and the CTA goes on to the common cluster barriers, which frees TMEM.
#include "pair_gemm.cuh"

namespace cg = cooperative_groups;

namespace b200 {

int sm_count();
bool rows_in_l2(int64_t D, int64_t H);
int pair_gate_up_values(const void* x, const void* gate, const float* bias, const void* up, void* packed,
                        float* values, int64_t M, int64_t D, int64_t H, int cf, cudaStream_t stream);
int twell_values_t2d(const void* packed, const float* values, const void* down, void* out, int64_t M,
                     int64_t D, int64_t H, int cf, void* workspace, size_t workspace_bytes,
                     cudaStream_t stream);

namespace {

namespace tm {

constexpr int kThreads = 352;
constexpr int kRows = 128;                 // tokens per CTA
constexpr int kRowBytes = kRows * 128;     // their 64-k stage
constexpr int kRing = 192 * 1024;          // shared memory of the stages

__device__ int g_error = 0;

__device__ __forceinline__ void give_up(int* abort_s, int code) {
  *(volatile int*)abort_s = 1;
  atomicExch(&g_error, code);
}

template <int STAGES>
struct Ring {
  uint64_t full[STAGES], empty[STAGES], done;
  uint64_t up_full[2], up_empty[2];  // VALUES: ranges of the up product
  uint32_t tmem;
  int abort;
};

// Barriers and TMEM; every thread of the cluster takes part in the cluster barrier that the caller
// waits for before it touches another CTA's shared memory.
template <int STAGES, int COLS>
__device__ __forceinline__ void set_up(Ring<STAGES>& r, int warp) {
  if (threadIdx.x == 0) {
#pragma unroll
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&r.full[s], 2);  // both producers
      mbar_init(&r.empty[s], 1);
    }
    mbar_init(&r.done, 1);
#pragma unroll
    for (int b = 0; b < 2; ++b) {
      mbar_init(&r.up_full[b], 1);
      mbar_init(&r.up_empty[b], 8);  // the epilogue warps
    }
    r.abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 2) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                 ::"r"(smem_u32(&r.tmem)), "r"(COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}

// One producer thread: `load(k, stage)` issues its copies of a k-step, `bytes` in all.
template <int STAGES, typename Load>
__device__ __forceinline__ void produce(Ring<STAGES>& r, int ksteps, uint32_t bytes, int code, Load load) {
  if (!ring_produce<STAGES>(r.full, r.empty, ksteps, bytes, load)) give_up(&r.abort, code);
}

// The MMA thread.
template <int STAGES, typename Step>
__device__ __forceinline__ void issue(Ring<STAGES>& r, int ksteps, int code, Step step) {
  if (ring_issue<STAGES>(r.full, r.empty, ksteps, step)) umma_commit(&r.done);
  else give_up(&r.abort, code);
}

template <int STAGES, int COLS>
__device__ __forceinline__ void free_tmem(Ring<STAGES>& r, int warp) {
  if (warp != 2) return;
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(r.tmem), "r"(COLS)
               : "memory");
}

// 32 columns of sums, added over the ranges in their order.
template <int RANGES, int COLS>
__device__ __forceinline__ void load_sums(uint32_t addr, float (&v)[32]) {
  tmem_ld32(addr, v);
#pragma unroll
  for (int r = 1; r < RANGES; ++r) {
    float w[32];
    tmem_ld32(addr + (uint32_t)(r * COLS), w);
#pragma unroll
    for (int c = 0; c < 32; ++c) v[c] += w[c];
  }
}

// The MMA thread of the form with fp32 hidden values where a quarter of D is more than kDrain k-steps or TMEM
// does not hold four ranges of both products: the gate product in RANGES ranges of k at TMEM column 0,
// the up product in ranges of kDrain k-steps that alternate between two accumulators at column 256, which the
// epilogue warps empty.
template <int STAGES, int NB, int RANGES>
__device__ __forceinline__ bool issue_values(Ring<STAGES>& r, int ksteps, uint64_t da0) {
  constexpr uint32_t kStage = kRowBytes + 2 * NB * 128, kIdesc = umma_idesc(kRows, NB);
  int s = 0, range = -1, next = 0;
  uint32_t phase = 0;
#pragma unroll 1
  for (int k = 0; k < ksteps; ++k) {
    const int up = k / pg::kDrain, b = up & 1;
    const bool up_first = k % pg::kDrain == 0;
    if (!mbar_wait(&r.full[s], phase)) return false;
    if (up_first && !mbar_wait(&r.up_empty[b], ((uint32_t)(up >> 1) & 1u) ^ 1u)) return false;
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const bool first = k == next;
    if (first) next = (++range + 1) * ksteps / RANGES;
    const uint64_t da = da0 + (uint32_t)s * (kStage >> 4), db = da + (kRowBytes >> 4);
#pragma unroll
    for (int kk = 0; kk < kStageK / 16; ++kk) {
      umma_bf16(r.tmem + (uint32_t)(range * NB), da + 2 * kk, db + 2 * kk, kIdesc, !first || kk > 0 ? 1u : 0u);
      umma_bf16(r.tmem + (uint32_t)(256 + b * NB), da + 2 * kk, db + (NB * 128 >> 4) + 2 * kk, kIdesc,
                !up_first || kk > 0 ? 1u : 0u);
    }
    umma_commit(&r.empty[s]);
    if ((k + 1) % pg::kDrain == 0 || k + 1 == ksteps) umma_commit(&r.up_full[b]);
    if (++s == STAGES) {
      s = 0;
      phase ^= 1u;
    }
  }
  umma_commit(&r.done);
  return true;
}

struct FirstArgs {
  const float* bias;      // bias16: 16-byte aligned
  int bias16;
  uint32_t* packed;
  int slab_w, row_words;
  __nv_bfloat16* hidden;  // [M][H]
  float* values;          // VALUES: instead of hidden, fp32 values in the slots of the slab [M][row_words]
  long long H;
  int wide;               // hidden rows are 32-byte aligned
  int M, ksteps, box;     // box: token rows per copy
  int keep_all;           // values past a slab's capacity still count in the product
  unsigned int* counts;   // stored entries of each 256 neurons, all tokens (one row tile), or null
  int64_t row_step;       // host: rows of x are every row_step-th token
};

// grid = (H / NB, ceil(M / 128)), cluster = 256 / NB along the neurons.
template <bool GATED, bool VALUES, bool DRAIN, int NB, int RANGES>
__global__ void __launch_bounds__(kThreads, 1)
first_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_g,
             const __grid_constant__ CUtensorMap map_u, const __grid_constant__ FirstArgs a) {
  constexpr int CL = kTileN / NB;
  constexpr int COLS = (GATED ? 2 : 1) * NB;
  constexpr int kStage = kRowBytes + COLS * 128;
  constexpr int STAGES = kRing / kStage > 8 ? 8 : kRing / kStage;
  constexpr int BLKS = NB / 64;  // 32-column blocks per epilogue warp
  constexpr int kTmem = DRAIN ? 512 : RANGES * COLS;
  // Four ranges of k (two where TMEM holds no more) stay apart and are added in fp32: a tensor core's
  // running sum loses bits with its length.  Stored gate values of N(0, 1) tokens that are not the rounded
  // 64-bit value, one range / four: D 1024 0.55 / 0.16 %, D 2048 1.07 / 0.33 %, D 4096 1.81 / 0.71 %.  The
  // pack of the same size splits D the same way, so its slab words are the same.
  static_assert(RANGES * (DRAIN ? 2 * NB : COLS) <= 512, "TMEM columns");
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  __shared__ __align__(8) Ring<STAGES> ring;
  __shared__ int count[2 * CL][kRows];  // stored entries by (rank, column half) and token

  cg::cluster_group cluster = cg::this_cluster();
  const int crank = (int)blockIdx.x % CL;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n0 = (int)blockIdx.x * NB, m0 = (int)blockIdx.y * kRows;
  cluster.barrier_arrive();
  set_up<STAGES, kTmem>(ring, warp);
  if (threadIdx.x == 0)
    for (int k = 0; k < 2 && k < a.ksteps; ++k) {
      tma_prefetch_2d(&map_g, k * kStageK, n0);
      if (GATED) tma_prefetch_2d(&map_u, k * kStageK, n0);
    }
  pdl_wait();

  uint32_t gw[BLKS][16];  // gate values as bf16 pairs, zero where nothing is stored
  uint32_t mask[BLKS];
  float u[DRAIN ? BLKS : 1][32] = {};
  int cnt = 0;
  bool ok = false;
  const int q = warp & 3, half = (warp - 3) >> 2;
  const int rl = q * 32 + lane, row = m0 + rl;
  const bool live = row < a.M;
  const uint32_t acc = ring.tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(half * (NB / 2));
  if (warp == 0) {
    if (elect_one())
      produce(ring, a.ksteps, COLS * 128, 1, [&](int k, int s) {
        unsigned char* b = smem + (size_t)s * kStage + kRowBytes;
        tma_load_2d(b, &map_g, k * kStageK, n0, &ring.full[s]);
        if (GATED) tma_load_2d(b + NB * 128, &map_u, k * kStageK, n0, &ring.full[s]);
      });
  } else if (warp == 1) {
    if (elect_one())
      produce(ring, a.ksteps, a.box * 128, 2, [&](int k, int s) {
        tma_load_2d(smem + (size_t)s * kStage, &map_x, k * kStageK, m0, &ring.full[s]);
      });
  } else if (warp == 2) {
    const uint64_t da0 = umma_desc(smem_u32(smem));
    const uint32_t tmem = ring.tmem;
    if (elect_one()) {
      if constexpr (DRAIN) {
        if (!issue_values<STAGES, NB, RANGES>(ring, a.ksteps, da0)) give_up(&ring.abort, 3);
      } else {
        issue(ring, a.ksteps, 3, [&, k = 0, range = -1, next = 0](bool, int s) mutable {
          const bool first = k++ == next;
          if (first) next = (++range + 1) * a.ksteps / RANGES;
          const uint64_t da = da0 + (uint32_t)s * (kStage >> 4), db = da + (kRowBytes >> 4);
#pragma unroll
          for (int kk = 0; kk < kStageK / 16; ++kk)
            umma_bf16(tmem + (uint32_t)(range * COLS), da + 2 * kk, db + 2 * kk, umma_idesc(kRows, COLS),
                      !first || kk > 0 ? 1u : 0u);
        });
      }
    }
  } else {
    if (DRAIN) {  // the up product, range by range
      ok = true;
      for (int r = 0; r * pg::kDrain < a.ksteps && ok; ++r) {
        ok = mbar_wait(&ring.up_full[r & 1], (uint32_t)(r >> 1) & 1u);
        ok = __all_sync(0xffffffffu, ok);
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
        for (int b = 0; b < BLKS && ok; ++b) {
          float w[32];
          tmem_ld32(acc + (uint32_t)(256 + (r & 1) * NB + b * 32), w);
#pragma unroll
          for (int c = 0; c < 32; ++c) u[b][c] += w[c];
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (lane == 0) mbar_arrive(&ring.up_empty[r & 1]);
      }
    }
    ok = mbar_wait(&ring.done, 0u) && (ok || !DRAIN);
    ok = __all_sync(0xffffffffu, ok);
    if (!ok) give_up(&ring.abort, 4);
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
    for (int b = 0; b < BLKS; ++b) {
      float v[32];
      load_sums<RANGES, DRAIN ? NB : COLS>(acc + (uint32_t)(b * 32), v);
      if (a.bias != nullptr) {
        const float* bp = a.bias + n0 + half * (NB / 2) + b * 32;
        if (a.bias16) {
#pragma unroll
          for (int c = 0; c < 8; ++c) {
            const float4 bv = __ldg(reinterpret_cast<const float4*>(bp) + c);
            v[4 * c] += bv.x;
            v[4 * c + 1] += bv.y;
            v[4 * c + 2] += bv.z;
            v[4 * c + 3] += bv.w;
          }
        } else {
#pragma unroll
          for (int c = 0; c < 32; ++c) v[c] += __ldg(bp + c);
        }
      }
      uint32_t m = 0;
#pragma unroll
      for (int c = 0; c < 32; ++c) m |= v[c] > 0.f ? 1u << c : 0u;
      mask[b] = live ? m : 0u;
      cnt += __popc(mask[b]);
#pragma unroll
      for (int p = 0; p < 16; ++p) gw[b][p] = pg::pack2(fmaxf(v[2 * p], 0.f), fmaxf(v[2 * p + 1], 0.f));
    }
  }
  if (warp == 0 && (VALUES || a.hidden != nullptr)) pdl_trigger();  // not for a contraction after a pack
  cluster.barrier_wait();  // every CTA of the cluster runs
  if (warp >= 3) {
#pragma unroll
    for (int r = 0; r < CL; ++r) *cluster.map_shared_rank(&count[2 * crank + half][rl], r) = cnt;
  }
  cluster.sync();
  if (a.counts != nullptr && warp == 3 && crank == 0) {
    int n = 0;
    for (int r = lane; r < a.M; r += 32) {
      int total = 0;
#pragma unroll
      for (int i = 0; i < 2 * CL; ++i) total += count[i][r];
      n += min(total, a.slab_w - 1);
    }
    n = __reduce_add_sync(0xffffffffu, n);
    if (lane == 0) a.counts[blockIdx.x / CL] = (unsigned int)n;
  }
  if (warp >= 3 && ok) {
    int slot = 0, total = 0;
#pragma unroll
    for (int i = 0; i < 2 * CL; ++i) {
      const int c = count[i][rl];
      if (i < 2 * crank + half) slot += c;
      total += c;
    }
    const int cap = a.slab_w - 1, tile = (int)blockIdx.x / CL;
    uint32_t* slab = a.packed + (size_t)row * a.row_words + (size_t)tile * a.slab_w;
    float* values = VALUES ? a.values + (size_t)row * a.row_words + (size_t)tile * a.slab_w : nullptr;
    if (crank == 0 && half == 0 && live) slab[0] = (uint32_t)total;
    __nv_bfloat16* out = a.hidden + (size_t)row * a.H + n0 + half * (NB / 2);
#pragma unroll
    for (int b = 0; b < BLKS; ++b) {
      if (total > cap) {  // values past the slab's capacity are not stored and leave the product too
        uint32_t m = mask[b];
        while (__popc(m) > max(cap - slot, 0)) m &= ~(0x80000000u >> __clz(m));
        mask[b] = m;
#pragma unroll
        for (int p = 0; p < 16 && !a.keep_all; ++p)
          gw[b][p] &= ((m >> (2 * p)) & 1u ? 0xFFFFu : 0u) | ((m >> (2 * p + 1)) & 1u ? 0xFFFF0000u : 0u);
      }
      const uint32_t col0 = (uint32_t)(n0 + half * (NB / 2) + b * 32), m = mask[b];
      if (VALUES && !DRAIN) {
        __syncwarp();
        load_sums<RANGES, COLS>(acc + (uint32_t)(NB + b * 32), u[0]);
      }
#pragma unroll
      for (int c = 0; c < 32; ++c)
        if ((m >> c) & 1u) {
          ++slot;
          slab[slot] = (col0 + c) | (c & 1 ? gw[b][c / 2] & 0xFFFF0000u : gw[b][c / 2] << 16);
          if (VALUES) values[slot] = (c & 1 ? pg::hi_f(gw[b][c / 2]) : pg::lo_f(gw[b][c / 2])) * u[DRAIN ? b : 0][c];
        }
      if (VALUES) {
      } else if (!GATED) {
        if (live && a.hidden != nullptr) pg::store64(out + b * 32, gw[b], a.wide);
      } else {
        float v[32];
        __syncwarp();
        load_sums<RANGES, COLS>(acc + (uint32_t)(NB + b * 32), v);
        uint32_t w[16];
#pragma unroll
        for (int p = 0; p < 16; ++p) {
          const uint32_t nz = pg::nonzero2(gw[b][p]);  // never touch u where nothing is stored
          w[p] = pg::mul2(gw[b][p], pg::pack2(v[2 * p], v[2 * p + 1]) & nz) & nz;
        }
        if (live) pg::store64(out + b * 32, w, a.wide);
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  free_tmem<STAGES, kTmem>(ring, warp);
}

// Owner's place of a 16-byte piece (0..3) of a token's 16 sums: pieces rotate with the row pair, so
// that eight lanes on eight rows reach all banks.
__device__ __forceinline__ float* sum_at(float* sums, int src, int row, int piece) {
  return sums + ((size_t)src * kRows + row) * 16 + ((piece ^ ((row >> 1) & 3)) << 2);
}

// grid = (D / ND * CL, ceil(M / 128)), cluster = CL along k.  map_d: the weights as they are stored, [H][D].
template <int ND, int CL>
__global__ void __launch_bounds__(kThreads, 1)
second_kernel(const __grid_constant__ CUtensorMap map_h, const __grid_constant__ CUtensorMap map_d,
              __nv_bfloat16* __restrict__ out, int M, int D, int ksteps, int box) {
  constexpr int PER = ND / CL / 16;             // 16-column groups per owner (1 or 2 or 4)
  constexpr int kSums = PER * CL * kRows * 64;  // bytes received: ND x 128 fp32
  constexpr int kStage = kRowBytes + ND * 128;
  constexpr int STAGES = (224 * 1024 - kSums) / kStage > 8 ? 8 : (224 * 1024 - kSums) / kStage;
  constexpr uint32_t kIdesc = umma_idesc(kRows, ND) | 1u << 16;
  static_assert(ND % (16 * CL) == 0, "an owner's columns are whole 16-column groups");
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  float* sums = reinterpret_cast<float*>(smem + (size_t)STAGES * kStage);  // [PER][CL][128][16]
  __shared__ __align__(8) Ring<STAGES> ring;

  cg::cluster_group cluster = cg::this_cluster();
  const int crank = (int)blockIdx.x % CL;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int c0 = (int)blockIdx.x / CL * ND, m0 = (int)blockIdx.y * kRows;
  const int k0 = crank * ksteps / CL, k1 = (crank + 1) * ksteps / CL;
  cluster.barrier_arrive();
  set_up<STAGES, ND>(ring, warp);
  pdl_wait();

  bool ok = false;
  const int q = warp & 3, half = (warp - 3) >> 2;
  if (warp == 0) {
    if (elect_one())
      produce(ring, k1 - k0, ND * 128, 5, [&](int k, int s) {
        unsigned char* b = smem + (size_t)s * kStage + kRowBytes;
#pragma unroll
        for (int i = 0; i < ND / 64; ++i)
          tma_load_2d(b + i * 8192, &map_d, c0 + i * 64, (k0 + k) * kStageK, &ring.full[s]);
      });
  } else if (warp == 1) {
    if (elect_one())
      produce(ring, k1 - k0, box * 128, 6, [&](int k, int s) {
        tma_load_2d(smem + (size_t)s * kStage, &map_h, (k0 + k) * kStageK, m0, &ring.full[s]);
      });
  } else if (warp == 2) {
    const uint64_t da0 = umma_desc(smem_u32(smem)), db0 = pg::desc_mn(smem_u32(smem) + kRowBytes);
    const uint32_t tmem = ring.tmem;
    if (elect_one())
      issue(ring, k1 - k0, 7, [&](bool first, int s) {
        const uint64_t da = da0 + (uint32_t)s * (kStage >> 4), db = db0 + (uint32_t)s * (kStage >> 4);
#pragma unroll
        for (int kk = 0; kk < kStageK / 16; ++kk)
          umma_bf16(tmem, da + 2 * kk, db + 128 * kk, kIdesc, !first || kk > 0 ? 1u : 0u);
      });
  } else {
    ok = mbar_wait(&ring.done, 0u);
    ok = __all_sync(0xffffffffu, ok);
    if (!ok) give_up(&ring.abort, 8);
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  }
  if (warp == 0) pdl_trigger();
  cluster.barrier_wait();  // every CTA of the cluster runs
  if (warp >= 3 && ok && m0 + q * 32 < M) {
    const int rl = q * 32 + lane;
    const uint32_t acc = ring.tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(half * (ND / 2));
#pragma unroll
    for (int b = 0; b < ND / 64; ++b) {
      float v[32];
      __syncwarp();
      tmem_ld32(acc + (uint32_t)(b * 32), v);
#pragma unroll
      for (int g = 0; g < 2 && m0 + rl < M; ++g) {
        const int group = half * (ND / 32) + b * 2 + g;  // of 16 columns
        float* dst = cluster.map_shared_rank(sums, group / PER) + (size_t)(group % PER) * CL * kRows * 16;
#pragma unroll
        for (int p = 0; p < 4; ++p)
          *reinterpret_cast<float4*>(sum_at(dst, crank, rl, p)) =
              make_float4(v[16 * g + 4 * p], v[16 * g + 4 * p + 1], v[16 * g + 4 * p + 2],
                          v[16 * g + 4 * p + 3]);
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  cluster.sync();
  free_tmem<STAGES, ND>(ring, warp);
  if (warp < 3 || ring.abort) return;
  const int et = threadIdx.x - 96, rl = et >> 1, row = m0 + rl;
  if (row >= M) return;
#pragma unroll
  for (int i = 0; i < PER; ++i) {
    float* mine = sums + (size_t)i * CL * kRows * 16;
    float v[8];
#pragma unroll
    for (int c = 0; c < 8; ++c) v[c] = 0.f;
#pragma unroll
    for (int r = 0; r < CL; ++r)
#pragma unroll
      for (int p = 0; p < 2; ++p) {
        const float4 u = *reinterpret_cast<const float4*>(sum_at(mine, r, rl, 2 * (et & 1) + p));
        v[4 * p] += u.x;
        v[4 * p + 1] += u.y;
        v[4 * p + 2] += u.z;
        v[4 * p + 3] += u.w;
      }
    *reinterpret_cast<uint4*>(out + (size_t)row * D + c0 + (crank * PER + i) * 16 + 8 * (et & 1)) =
        make_uint4(pg::pack2(v[0], v[1]), pg::pack2(v[2], v[3]), pg::pack2(v[4], v[5]),
                   pg::pack2(v[6], v[7]));
  }
}

template <typename Kernel, typename... Args>
int launch_cluster(const char* fn, Kernel kern, dim3 grid, int cluster, size_t smem, size_t (&granted)[64],
                   cudaStream_t stream, Args... args) {
  if (int rc = ensure_dynamic_smem(kern, smem, granted, fn)) return rc;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(kThreads, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)cluster;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = add_pdl_attribute(attr, 1);
  cudaError_t e = cudaLaunchKernelEx(&cfg, kern, args...);
  if (e != cudaSuccess) return fail(B200_ECUDA, "%s: launch: %s", fn, cudaGetErrorString(e));
  return B200_OK;
}

template <bool GATED, bool VALUES, int NB, bool DRAIN = VALUES && NB == 128>
int launch_first(const void* x, const void* g, const void* u, FirstArgs a, int64_t D, cudaStream_t stream) {
  constexpr int RANGES = GATED ? 256 / NB : 4;
  constexpr int kStage = kRowBytes + (GATED ? 2 : 1) * NB * 128;
  constexpr int STAGES = kRing / kStage > 8 ? 8 : kRing / kStage;
  CUtensorMap mx, mg, mu;
  if (int rc = make_map(&mx, x, a.M, D, a.box, kStageK, a.row_step)) return rc;
  if (int rc = make_map(&mg, g, a.H, D, NB)) return rc;
  if (int rc = make_map(&mu, u, a.H, D, NB)) return rc;
  static size_t granted[64] = {0};
  return launch_cluster("gate and up tiles", first_kernel<GATED, VALUES, DRAIN, NB, RANGES>,
                        dim3((unsigned)(a.H / NB), (unsigned)((a.M + kRows - 1) / kRows), 1), kTileN / NB,
                        (size_t)STAGES * kStage + 1024, granted, stream, mx, mg, mu, a);
}

template <int ND, int CL>
int launch_second(const void* hidden, const void* down, void* out, int64_t M, int64_t D, int64_t H,
                  int box, cudaStream_t stream) {
  constexpr int kSums = ND * kRows * 4;
  constexpr int kStage = kRowBytes + ND * 128;
  constexpr int STAGES = (224 * 1024 - kSums) / kStage > 8 ? 8 : (224 * 1024 - kSums) / kStage;
  CUtensorMap mh, md;
  if (int rc = make_map(&mh, hidden, M, H, box)) return rc;
  if (int rc = make_map(&md, down, H, D, 64)) return rc;
  static size_t granted[64] = {0};
  return launch_cluster("down tiles", second_kernel<ND, CL>,
                        dim3((unsigned)(D / ND * CL), (unsigned)((M + kRows - 1) / kRows), 1), CL,
                        (size_t)STAGES * kStage + kSums + 1024, granted, stream, mh, md,
                        static_cast<__nv_bfloat16*>(out), (int)M, (int)D, (int)(H / kStageK),
                        box);
}

}  // namespace tm

}  // namespace

namespace {

// CTAs in clusters of four that are resident at once (a GPC's SMs are no multiple of four).
int64_t fours() { return (sm_count() / 4 - 4) * 4; }
int64_t row_tiles(int64_t M) { return (M + tm::kRows - 1) / tm::kRows; }
int token_box(int64_t M) { return M < tm::kRows ? (int)((M + 7) / 8 * 8) : tm::kRows; }

}  // namespace

// Which calls of the fused MLPs run here.  Up to 32 tokens the gathers touch few rows (D 2048, H 8192, 32
// tokens, 0.5 % / 2 % 17 / 24 us against 24).  Beyond, a call cannot know its density: the line lies where the
// tiles are level with the gathers at 1 %, and gated layers whose rows come from HBM wait until they are level
// at 0.5 %.  For wide layers that is later, as the tiles stream all of up and
// down.  us per layer under graph replay, weights from HBM, gathers at 0.5 / 1 / 2 % -> tiles (any density):
//   gated    D 1024, H 4096:   33 tokens 13.4 / 14.0 / 15.9 -> 13.3;  128 tokens 16.9 / 19.0 / 23.3 -> 15.1
//            D 2048, H 5632:   33 tokens 17.7 / 19.9 / 22.0 -> 19.7;  128 tokens 22.4 / 26.6 / 35.0 -> 21.9
//            D 2048, H 8192:   33 tokens 18.9 / 21.1 / 25.0 -> 24.4 (not taken);  40 tokens 20.5 / 23.6 / 29.7
//                              -> 24.6;  128 tokens 25.5 / 31.9 / 43.8 -> 26.9
//            D 2048, H 11008:  64 tokens 25.9 / 30.4 / 38.6 -> 33.4 (not taken);  80 tokens 29.7 / 37.7 / 52.3
//                              -> 33.8
//            D 4096, H 16384:  64 tokens 60.5 / 76.8 / 108 -> 75.3 (not taken);  80 tokens 72 / 102 / 163 -> 76
//   plain    D 2048, H 11008:  33 tokens 21.4 / 23.2 / 25.8 -> 24.9;  64 tokens 23.0 / 26.0 / 30.3 -> 25.5
//            D 4096, H 16384:  64 tokens 43.1 / 48.2 / 57.7 -> 54.1 (not taken);  96 tokens 49.0 / 58.4 / 76.1
//                              -> 56.3
// and while the first launch fits one wave: against the pairs of SMs, D 1024, H 4096, 256 tokens 35 -> 17, 512
// tokens 32 -> 23; D 2048, H 5632, 384 tokens 47 -> 34; H 8192, 256 tokens 48 -> 36; D 4096, H 16384, 128
// tokens 91 -> 80.  In two waves the form is level with the pairs at best (H 11008, 200 tokens 49 -> 54).
//
// One row tile at H 8704 to 9472 stays with the gathers (or the pairs): its pack adds four ranges of D, of
// which the accumulators of 128 neurons hold two.
static bool tiles_fit(int64_t M, int64_t D, int64_t H, bool gated) {
  if (M < 33 || M > 512 || D > 4096 || H < 2048) return false;
  if (gated && M <= tm::kRows && H / 64 > fours() && H / 64 <= sm_count()) return false;
  return row_tiles(M) * (H / 128) <= sm_count();
}

bool tile_mlp_serves(int64_t M, int64_t D, int64_t H, bool gated) {
  const int64_t from = gated ? (D * H <= (int64_t)12 << 20 ? 33 : D * H <= (int64_t)1 << 24 ? 40 : 80)
                             : (D * H <= (int64_t)1 << 25 ? 33 : 96);
  return M >= from && tiles_fit(M, D, H, gated);
}

// Slabs and hidden values ([M, H] bf16, 16-byte aligned); keep_all: of every gate positive, not only of
// the stored ones.  values (gated): instead of hidden, their fp32 hidden values in the slots of the slabs.
int tile_first(bool gated, const void* x, const void* gate, const float* bias, const void* up,
               void* packed, void* hidden, float* values, int64_t M, int64_t D, int64_t H, int cf,
               bool keep_all, cudaStream_t stream) {
  tm::FirstArgs a = {};
  a.bias = bias;
  a.bias16 = aligned16(bias);
  a.packed = static_cast<uint32_t*>(packed);
  a.slab_w = kTileN / cf;
  a.row_words = (int)(H / kTileN) * a.slab_w;
  a.hidden = static_cast<__nv_bfloat16*>(hidden);
  a.values = values;
  a.H = H;
  a.wide = (reinterpret_cast<uintptr_t>(hidden) & 31u) == 0;
  a.M = (int)M;
  a.ksteps = (int)(D / kStageK);
  a.box = token_box(M);
  a.row_step = 1;
  a.keep_all = keep_all;
  // 64 neurons per CTA while that is one wave: 128 tokens, D 2048, H 8192 16.5 against 21 us; the
  // accumulators of 128 neurons cost twice the MMAs per step.
  if (row_tiles(M) * (H / 64) <= fours())
    return values != nullptr ? (D <= 2048 ? tm::launch_first<true, true, 64>(x, gate, up, a, D, stream)
                                          : tm::launch_first<true, true, 64, true>(x, gate, up, a, D, stream))
           : gated           ? tm::launch_first<true, false, 64>(x, gate, up, a, D, stream)
                             : tm::launch_first<false, false, 64>(x, gate, gate, a, D, stream);
  return values != nullptr ? tm::launch_first<true, true, 128>(x, gate, up, a, D, stream)
         : gated           ? tm::launch_first<true, false, 128>(x, gate, up, a, D, stream)
                           : tm::launch_first<false, false, 128>(x, gate, gate, a, D, stream);
}

// Whether a pack runs here: 33 to 256 tokens while the grid is one wave, and 17 to 32 tokens where the
// four-way split over a cluster is more than one.  us, split-k (or pairs of SMs) / here, weights from HBM:
//   33 to 128 tokens   D 1024, H 4096 10.9 / 7.4;  D 2048, H 2048 12.5 / 10.5;  H 5632 13.9 / 11.1;
//                      H 8192 15.5 / 11.6;  H 11008 18.6 / 14.7;  D 4096, H 4096 16.9 / 16.8;  H 16384 34.5 / 29.5
//   256 tokens         D 1024, H 4096 12.3 / 7.9;  D 2048, H 4096 14.0 / 11.0;  H 8192 17.7 / 13.8;
//                      two waves: H 11008 18.7 / 25.3
//   32 tokens          D 2048, H 5632 8.8 / 10.9;  H 8192 10.5 / 11.5;  two waves of the split: H 11008
//                      17.8 / 14.5;  D 4096, H 16384 32.7 / 29.4
bool tile_pack_serves(int64_t M, int64_t H) {
  if (M <= 32) return M > 16 && H / 64 > fours() && H / 128 <= sm_count();
  return M <= 256 && row_tiles(M) * (H / 128) <= sm_count();
}

// Slabs only.
int tile_pack(const void* x, const void* w, const float* bias, void* packed, int64_t M, int64_t D,
              int64_t H, int cf, cudaStream_t stream) {
  tm::FirstArgs a = {};
  a.bias = bias;
  a.bias16 = aligned16(bias);
  a.packed = static_cast<uint32_t*>(packed);
  a.slab_w = kTileN / cf;
  a.row_words = (int)(H / kTileN) * a.slab_w;
  a.H = H;
  a.M = (int)M;
  a.ksteps = (int)(D / kStageK);
  a.box = token_box(M);
  a.row_step = 1;
  if (row_tiles(M) * (H / 64) <= fours())
    return tm::launch_first<false, false, 64>(x, w, w, a, D, stream);
  return tm::launch_first<false, false, 128>(x, w, w, a, D, stream);
}

// Slabs of kSampleTokens tokens spread evenly over the M of a call, and their stored entries by 256 neurons.
int tile_sample(const void* x, const void* w, const float* bias, void* packed, unsigned int* counts,
                int64_t M, int64_t D, int64_t H, int cf, cudaStream_t stream) {
  tm::FirstArgs a = {};
  a.bias = bias;
  a.bias16 = aligned16(bias);
  a.packed = static_cast<uint32_t*>(packed);
  a.slab_w = kTileN / cf;
  a.row_words = (int)(H / kTileN) * a.slab_w;
  a.H = H;
  a.M = kSampleTokens;
  a.ksteps = (int)(D / kStageK);
  a.box = token_box(a.M);
  a.row_step = M / kSampleTokens;
  a.counts = counts;
  if (H / 64 <= fours()) return tm::launch_first<false, false, 64>(x, w, w, a, D, stream);
  return tm::launch_first<false, false, 128>(x, w, w, a, D, stream);
}

// out[M, D] = hidden[M, H] down with down [H, D] as it is stored.
int tile_second(const void* hidden, const void* down, void* out, int64_t M, int64_t D, int64_t H,
                cudaStream_t stream) {
  const int box = token_box(M);
  // As with the neurons, and k in four slices: 128 tokens, D 2048 12.5 (64 columns) against
  // 16 us (128); 256 tokens 35 against 21.  Clusters of eight fit half the GPU at once (21 us).
  if (row_tiles(M) * (D / 64) * 4 <= fours())
    return tm::launch_second<64, 4>(hidden, down, out, M, D, H, box, stream);
  if (row_tiles(M) * (D / 128) * 4 <= fours())
    return tm::launch_second<128, 4>(hidden, down, out, M, D, H, box, stream);
  return tm::launch_second<128, 2>(hidden, down, out, M, D, H, box, stream);
}

// High precision below the sizes of pair_mlp_serves: gate and up as tensor-core products, here or on pairs
// of SMs, and the down product gathered along the stored entries with fp32 hidden values (half the rows
// that gathering both reads, and no partial sums of the up product).  The lines lie as above.  us per layer
// under graph replay, pack + gathers -> this form, at 0.5 / 1 / 2 % density:
//   D 1024, H 4096   33 tokens 13.3 / 13.9 / 15.5 -> 13.3 / 13.7 / 14.9;  257 tokens 23 / 28 / 35 -> 20 / 21 / 23;
//                    1500 tokens 43 / 54 / 79 -> 50 / 56 / 67;  4000 tokens 82 / 110 / 166 -> 92 / 104 / 131
//   D 2048, H 5632   48 tokens 19.3 / 21.3 / 25.0 -> 21.2 / 22.2 / 24.2;  160 tokens 28 / 35 / 49 -> 30 / 34 / 41
//   D 2048, H 8192   64 tokens 20.9 / 24.2 / 29.8 -> 24.3 / 26.5 / 29.5 (not taken);  96 tokens 24.3 / 29.5 / 40.5
//                    -> 26.6 / 29.7 / 35.2;  257 tokens 39 / 51 / 70 -> 47 / 52 / 60 (not taken: pairs of SMs
//                    that are mostly padding);  777 tokens 78 / 103 / 161 -> 80 / 90 / 118;  4000 tokens 298 / 411 /
//                    660 -> 290 / 345 / 439
//   D 2048, H 11008  160 tokens 43 / 57 / 85 -> 51 / 55 / 63;  257 tokens 53 / 67 / 95 -> 69 / 75 / 87 (not taken);  400 tokens 68 / 95 / 147 -> 73 / 82 / 98
//   D 4096, H 16384  48 tokens 55 / 67 / 94 -> 64 / 70 / 78 (not taken);  64 tokens 57 / 70 / 97 -> 65 / 70 / 78;
//                    200 tokens 105 / 157 / 256 -> 93 / 108 / 139
bool values_mlp_serves(int64_t M, int64_t D, int64_t H) {
  if (D > 4096 || H < 2048 || M * D * H >= (int64_t)1 << 36) return false;
  if (M >= 160) return !(M > 256 && M < 320 && D * H >= (int64_t)1 << 24 && rows_in_l2(D, H));
  const int64_t from = D * H <= (int64_t)1 << 23 ? 33 : D * H <= (int64_t)12 << 20 ? 48 : rows_in_l2(D, H) ? 96 : 64;
  return M >= from && tiles_fit(M, D, H, true);
}

// values: [M, H / cf] fp32, 16-byte aligned.
int values_mlp(const void* x, const void* gate, const float* bias, const void* up, const void* down,
               void* packed, void* out, int64_t M, int64_t D, int64_t H, int cf, void* workspace,
               size_t workspace_bytes, float* values, cudaStream_t stream) {
  const int rc = tiles_fit(M, D, H, true)
                     ? tile_first(true, x, gate, bias, up, packed, nullptr, values, M, D, H, cf, false, stream)
                     : pair_gate_up_values(x, gate, bias, up, packed, values, M, D, H, cf, stream);
  if (rc) return rc;
  return twell_values_t2d(packed, values, down, out, M, D, H, cf, workspace, workspace_bytes, stream);
}

int tile_mlp(bool gated, const void* x, const void* gate, const float* bias, const void* up,
             const void* down, void* packed, void* out, int64_t M, int64_t D, int64_t H, int cf,
             void* hidden, cudaStream_t stream) {
  if (int rc = tile_first(gated, x, gate, bias, up, packed, hidden, nullptr, M, D, H, cf, false, stream)) return rc;
  return tile_second(hidden, down, out, M, D, H, stream);
}

// Error word raised by a bounded wait that gave up (0 = none).  Reads and clears it; synchronises.
int tile_mlp_status() {
  int v = 0, zero = 0;
  if (cudaMemcpyFromSymbol(&v, tm::g_error, sizeof(int)) != cudaSuccess) return -1;
  if (v != 0) cudaMemcpyToSymbol(tm::g_error, &zero, sizeof(int));
  return v;
}

}  // namespace b200
