// The fused MLPs on the paired tensor-core GEMM (pair_gemm.cuh) for calls of more than a few
// dozen tokens: gate GEMM with the pack epilogue, up GEMM whose epilogue multiplies by the slab
// pattern, down GEMM over the resulting hidden matrix.
#include <initializer_list>

#include "pair_gemm.cuh"

namespace b200 {

int sm_count();
bool tile_pack_serves(int64_t M, int64_t H);
int tile_sample(const void* x, const void* w, const float* bias, void* packed, unsigned int* counts,
                int64_t M, int64_t D, int64_t H, int cf, cudaStream_t stream);
int twell_t2d_launch(bool gated, bool hp, const void* x, const void* packed, const void* up,
                     const void* down, void* out, int64_t M, int64_t D, int64_t H, int cf,
                     void* workspace, size_t workspace_bytes, int sm_count, cudaStream_t stream,
                     const unsigned char* skip_rows, const FusedAr* fused_ar, const RunIf& run_if);

namespace {

constexpr int64_t kHiddenBytes = (int64_t)1 << 30;  // hidden matrix of one row chunk

// Rows of all chunks but the last: whole tiles within kHiddenBytes and, where the caller sets it,
// max_rows.
int64_t chunk_rows(int64_t M, int64_t H, int terms, int64_t max_rows) {
  int64_t most = kHiddenBytes / (H * 2 * terms) / pg::kTile * pg::kTile;
  if (max_rows > 0 && max_rows < most)
    most = max_rows < pg::kTile ? pg::kTile : max_rows / pg::kTile * pg::kTile;
  return M < most ? M : most;
}

size_t align256(size_t v) { return (v + 255) & ~(size_t)255; }

// Largest split-tile buffer of the three products of a call of `rows` rows.
size_t mlp_part_bytes(int64_t rows, int64_t D, int64_t H, int terms) {
  const int64_t mt = (rows + pg::kTile - 1) / pg::kTile, slots = sm_count() / 2;
  const size_t a = pg::part_bytes(mt * (H / pg::kTile), (int)(D / kStageK), slots, false);
  const size_t b = pg::part_bytes(mt * (D / pg::kTile), (int)(H * terms / kStageK), slots, true);
  return a > b ? a : b;
}

pg::Args base_args(int64_t rows, int64_t n, int64_t k) {
  pg::Args a = {};
  a.rows = (int)rows;
  a.n_tiles = (int)(n / pg::kTile);
  a.ksteps = (int)((k + kStageK - 1) / kStageK);
  a.seg_ksteps = a.second_mt = 1 << 30;
  return a;
}

int aligned32(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 31u) == 0; }

// The contraction workspace's zero-filled counters, or null.
unsigned int* split_counters(void* workspace, size_t workspace_bytes) {
  return workspace != nullptr && workspace_bytes >= 16384 ? static_cast<unsigned int*>(workspace)
                                                          : nullptr;
}

}  // namespace

// Slabs of relu(x W^T + bias); `dense`: also the stored values as an [M, H] matrix.  entries: counter of stored entries or null.
int pair_pack(const void* x, const void* w, const float* bias, void* packed, void* dense, int64_t M,
              int64_t D, int64_t H, int cf, unsigned int* entries, const SplitRoom& room,
              cudaStream_t stream) {
  pg::Args a = base_args(M, H, D);
  a.bias = bias;
  a.bias16 = aligned16(bias);
  a.entries = entries;
  a.slab_p = static_cast<uint32_t*>(packed);
  a.slab_w = kTileN / cf;
  a.row_words = (int)(H / kTileN) * a.slab_w;
  pg::give_room(a, room);
  const pg::Operand ox = {x, M, D}, ow = {w, H, D};
  if (dense == nullptr)
    return pg::launch<pg::kPack, false, false>("b200_twell_pack", ox, ox, ow, ow, a, M, sm_count(),
                                               stream);
  a.out = static_cast<__nv_bfloat16*>(dense);
  a.ld = H;
  a.wide = aligned32(dense);
  return pg::launch<pg::kPackDense, false, false>("b200_twell_pack", ox, ox, ow, ow, a, M,
                                                  sm_count(), stream);
}

// hidden[M, 3 H] = gate values of the slabs times x up^T on their pattern, as three bf16 terms.
int pair_up(const void* x, const void* packed, const void* up, void* hidden, int64_t M, int64_t D,
            int64_t H, int cf, const RunIf& run_if, const SplitRoom& room, cudaStream_t stream) {
  pg::Args a = base_args(M, H, D);
  a.run_if = run_if;
  a.slab_p = const_cast<uint32_t*>(static_cast<const uint32_t*>(packed));
  a.slab_w = kTileN / cf;
  a.row_words = (int)(H / kTileN) * a.slab_w;
  a.out = static_cast<__nv_bfloat16*>(hidden);
  a.ld = 3 * H;
  a.wide = aligned32(hidden);
  pg::give_room(a, room);
  const pg::Operand ox = {x, M, D}, ou = {up, H, D};
  return pg::launch<pg::kMulHp, false, false>("up product", ox, ox, ou, ou, a, M, sm_count(), stream);
}

// out[M, D] = hidden[M, terms * H] [down; down; ...] with down [H, D] as it is stored.
int pair_down(const void* hidden, int terms, const void* down, void* out, int64_t M, int64_t D,
              int64_t H, const RunIf& run_if, const SplitRoom& room, cudaStream_t stream) {
  pg::Args a = base_args(M, D, terms * H);
  a.run_if = run_if;
  a.seg_ksteps = (int)(H / kStageK);
  a.out = static_cast<__nv_bfloat16*>(out);
  a.ld = D;
  a.wide = aligned32(out);
  pg::give_room(a, room);
  const pg::Operand oh = {hidden, M, terms * H}, od = {down, D, H};
  return pg::launch<pg::kStore, false, true>("down product", oh, oh, od, od, a, M, sm_count(),
                                             stream);
}

// Slabs and hidden matrix in one launch: the gate and up products of a tile follow one another in
// the two accumulators, and the pack epilogue of the first runs under the MMAs of the second.
// keep_all: hidden values are computed from every gate positive, not only from the stored ones.
// run_if: slabs in any case, the hidden matrix where the dense form runs.
int pair_gate_up(const void* x, const void* gate, const float* bias, const void* up, void* packed,
                 void* hidden, int64_t M, int64_t D, int64_t H, int cf, bool keep_all,
                 cudaStream_t stream, const RunIf& run_if = {nullptr, 0u, 0, nullptr}) {
  pg::Args a = base_args(M, H, D);
  a.run_if = run_if;
  a.bias = bias;
  a.bias16 = aligned16(bias);
  a.keep_all = keep_all;
  a.slab_p = static_cast<uint32_t*>(packed);
  a.slab_w = kTileN / cf;
  a.row_words = (int)(H / kTileN) * a.slab_w;
  a.out = static_cast<__nv_bfloat16*>(hidden);
  a.ld = H;
  a.wide = aligned32(hidden);
  const pg::Operand ox = {x, M, D}, og = {gate, H, D}, ou = {up, H, D};
  return pg::launch<pg::kGateUp, false, false>("gate and up products", ox, ox, og, ou, a, M,
                                               sm_count(), stream);
}

// The same in high precision: fp32 hidden values in the slots of the slabs (values: [M][H / cf]).
int pair_gate_up_values(const void* x, const void* gate, const float* bias, const void* up, void* packed,
                        float* values, int64_t M, int64_t D, int64_t H, int cf, cudaStream_t stream) {
  pg::Args a = base_args(M, H, D);
  a.bias = bias;
  a.bias16 = aligned16(bias);
  a.slab_p = static_cast<uint32_t*>(packed);
  a.slab_w = kTileN / cf;
  a.row_words = (int)(H / kTileN) * a.slab_w;
  a.values = values;
  const pg::Operand ox = {x, M, D}, og = {gate, H, D}, ou = {up, H, D};
  return pg::launch<pg::kGateUpHp, false, false>("gate and up products", ox, ox, og, ou, a, M,
                                                 sm_count(), stream);
}

// Up and down rows together stay in L2, where a gathered entry is cheaper.
bool rows_in_l2(int64_t D, int64_t H) { return 4 * H * D <= (int64_t)100 << 20; }

namespace {

// From this many tokens on the products are dense.  Measured under graph replay with weights from
// HBM, us per layer, gather form at 0.5 % / 1 % / 2 % density -> dense form (any density):
//   D 1024, H 4096:   256 tokens 25 / 29 / 36 -> 34;  320 tokens 33 / 38 / 48 -> 35;
//                     800 tokens 37 / 46 / 63 -> 39;  1200 tokens 43 / 55 / 77 -> 54
//   D 2048, H 8192:   128 tokens 30 / 37 / 49 -> 50;  160 tokens 46 / 57 / 80 -> 50;
//                     512 tokens 68 / 92 / 135 -> 57;  800 tokens 77 / 109 / 169 -> 92
//   D 2048, H 11008:  256 tokens 61 / 77 / 107 -> 54;  300 tokens 63 / 82 / 123 -> 82
//   D 4096, H 16384:  64 tokens - / 91 / - -> 93;  96 tokens 88 / 122 / 182 -> 95
// The call cannot know its density: the lines lie where the dense form is level or ahead at 1 %.  At
// 0.5 % it is up to 1.3 times slower where the tiles just exceed a wave (300 tokens at H 11008,
// 800 at H 8192, 1200 at H 4096), and level or ahead elsewhere.
int64_t dense_from(int64_t D, int64_t H) {
  return D * H <= (int64_t)1 << 23 ? 320 : rows_in_l2(D, H) ? 160 : 96;
}

}  // namespace

// Which calls of the fused MLPs take this form.  High precision pays three down products, so it
// needs a larger call; the non-gated MLP saves only half as much (600 tokens, D 1024, H 4096, gathers at
// 0.5 % / 2 % -> dense 21 / 30 -> 31; 300 tokens, D 2048, H 8192 33 / 53 -> 44).
bool pair_mlp_serves(int64_t M, int64_t D, int64_t H, bool gated, bool hp) {
  if (H < 2048) return false;  // few entries per token: nothing to gain
  if (hp) return M * D * H >= (int64_t)1 << 36;
  return M >= (gated ? 1 : 2) * dense_from(D, H);
}

// Which bf16 calls let the device choose between the dense and the gather form of the up and down products
// by their stored entries.  A gated call asks a sample, 128 tokens spread over it (13 us of one-SM tiles
// before the others, and contraction CTAs that return at once, 3 us); a non-gated one has its gate product
// count (a 4-byte memset and the contraction, some 9 us).  us at 0.1 / 0.2 / 0.5 / 1 / 2 % density, dense
// always -> asking:
//   gated      D 2048, H 8192,   9000 tokens 685 / 685 / 682 / 708 / 704 -> 420 / 486 / 646 / 699 / 718;
//                               16384 tokens 1216 / 1218 / 1220 / 1226 / 1236 -> 723 / 869 / 1134 / 1216 / 1237
//              D 2048, H 11008,  6000 tokens 606 / 633 / 617 / 582 / 664 -> 342 / 533 / 590 / 644 / 645
//   non-gated  D 2048, H 8192,  12000 tokens 598 / 613 / 606 / 653 / 629 -> 453 / 467 / 575 / 609 / 617
// Below 1.5 x 2^36 multiply-adds asking costs 5 to 10 % from 0.7 % on and saves at 0.2 % and less only (gated,
// H 8192, 4500 tokens 337 / 320 / 339 / 330 / 327 -> 240 / 272 / 365 / 360 / 368): dense always.
static bool asks(int64_t m, int64_t D, int64_t H, bool gated) {
  if (m * D * H < (int64_t)3 << 35) return false;
  return !gated || (m > 4096 && rows_in_l2(D, H) && H / kTileN <= kSampleWords);
}

// Stored entries per token up to which the gather form is the faster one.  Measured (D 2048, H 8192) in high
// precision: up + down 104 ns per token dense and 0.8 ns per entry gathered; D 4096, H 16384 (rows from HBM
// as well): 382 ns against 2.7 ns.  bf16: see asks().
static int64_t gather_entries(int64_t D, int64_t H, bool gated, bool hp) {
  if (hp) return H / (rows_in_l2(D, H) ? 64 : 112);
  return H / (gated ? 180 : rows_in_l2(D, H) ? 160 : 224);
}

static unsigned int clamp_limit(int64_t limit) {
  return (unsigned int)(limit < 0x7fffffff ? limit : 0x7fffffff);
}

size_t pair_part_bytes(int64_t M, int64_t D, int64_t H) { return mlp_part_bytes(M, D, H, 1); }

// The split-tile buffer of a chunked call: which tiles are cut depends on their number, so the
// shorter last chunk often needs more room than a full one.
static size_t chunks_part_bytes(int64_t M, int64_t rows, int64_t D, int64_t H, int terms) {
  const size_t full = mlp_part_bytes(rows, D, H, terms);
  const size_t last = M % rows != 0 ? mlp_part_bytes(M % rows, D, H, terms) : 0;
  return full > last ? full : last;
}

// 240 bytes of it take a 16-byte aligned scratch to the 256 bytes at which its parts begin (rows of
// sums are written 32 bytes at a time).
size_t pair_mlp_scratch_bytes(int64_t M, int64_t D, int64_t H, bool hp, int64_t max_rows) {
  const int terms = hp ? 3 : 1;
  const int64_t rows = chunk_rows(M, H, terms, max_rows);
  return 240 + align256((size_t)rows * H * 2 * terms) + 256 + chunks_part_bytes(M, rows, D, H, terms);
}

// workspace: the contraction workspace (its zero-filled counters; may be null).
int pair_mlp(bool gated, bool hp, const void* x, const void* gate, const float* bias,
             const void* up, const void* down, void* packed, void* out, int64_t M, int64_t D,
             int64_t H, int cf, void* workspace, size_t workspace_bytes, void* scratch,
             int64_t max_rows, cudaStream_t stream) {
  const int terms = hp ? 3 : 1;
  const int64_t rows = chunk_rows(M, H, terms, max_rows);
  const int64_t row_words = H / cf;
  scratch = reinterpret_cast<void*>(align256(reinterpret_cast<uintptr_t>(scratch)));
  unsigned char* p = static_cast<unsigned char*>(scratch) + align256((size_t)rows * H * 2 * terms);
  unsigned int* entries = reinterpret_cast<unsigned int*>(p);
  const SplitRoom room = {reinterpret_cast<float*>(p + 256), chunks_part_bytes(M, rows, D, H, terms),
                          split_counters(workspace, workspace_bytes)};
  for (int64_t r0 = 0; r0 < M; r0 += rows) {
    const int64_t m = M - r0 < rows ? M - r0 : rows;
    const void* xc = static_cast<const __nv_bfloat16*>(x) + r0 * D;
    void* pc = static_cast<uint32_t*>(packed) + r0 * row_words;
    void* oc = static_cast<__nv_bfloat16*>(out) + r0 * D;
    if (!hp && !asks(m, D, H, gated)) {
      if (int rc = gated ? pair_gate_up(xc, gate, bias, up, pc, scratch, m, D, H, cf, false, stream)
                         : pair_pack(xc, gate, bias, pc, scratch, m, D, H, cf, nullptr, room, stream))
        return rc;
      if (int rc = pair_down(scratch, 1, down, oc, m, D, H, {nullptr, 0u, 0, nullptr}, room, stream)) return rc;
      continue;
    }
    const int64_t per_token = gather_entries(D, H, gated, hp);
    if (!hp && gated) {
      // the sample's slabs lie where the hidden values will be
      const RunIf ask = {entries, clamp_limit(kSampleTokens * per_token), (int)(H / kTileN), entries + kSampleWords};
      const RunIf run_if = {ask.verdict, 0u, 0, nullptr};
      if (int rc = tile_sample(xc, gate, bias, scratch, entries, m, D, H, cf, stream)) return rc;
      if (int rc = pair_gate_up(xc, gate, bias, up, pc, scratch, m, D, H, cf, false, stream, ask)) return rc;
      if (int rc = pair_down(scratch, 1, down, oc, m, D, H, run_if, room, stream)) return rc;
      if (int rc = twell_t2d_launch(true, true, xc, pc, up, down, oc, m, D, H, cf, workspace,
                                    workspace_bytes, sm_count(), stream, nullptr, nullptr, run_if))
        return rc;
      continue;
    }
    const RunIf run_if = {entries, clamp_limit(m * per_token), 0, nullptr};
    if (cudaMemsetAsync(entries, 0, sizeof(unsigned int), stream) != cudaSuccess)
      return fail(B200_ECUDA, "fused MLP: cudaMemsetAsync failed");
    pdl_suppressed() = true;  // its predecessor is the memset
    const int rc = pair_pack(xc, gate, bias, pc, gated ? nullptr : scratch, m, D, H, cf, entries, room, stream);
    pdl_suppressed() = false;
    if (rc) return rc;
    if (gated)
      if (int rc = pair_up(xc, pc, up, scratch, m, D, H, cf, run_if, room, stream)) return rc;
    if (int rc = pair_down(scratch, terms, down, oc, m, D, H, run_if, room, stream)) return rc;
    // fp32 products, as the dense form does not round them one by one either
    if (int rc = twell_t2d_launch(gated, true, xc, pc, up, down, oc, m, D, H, cf, workspace,
                                  workspace_bytes, sm_count(), stream, nullptr, nullptr, run_if))
      return rc;
  }
  return B200_OK;
}

// ---- hybrid training operator --------------------------------------------------------------------
namespace {

// Overflow bookkeeping of one call, zero-filled before it.
struct RowState {
  int n_tail;       // rows taken out of the slabs
  int n_over;       // rows with an overflowed tile
  int dropped;      // entries lost to the slabs' capacity
  unsigned int done;
  unsigned long long nnz;
};

// Forward (BWD = false): a warp per row adds up the count words; the block that finishes last
// writes l0 and the lost entries, and lists the first `cap` overflowed rows in ascending order.
// Backward: the listed rows are those whose count words carry the sign bit.
// row_slot[r]: place of row r in the list, else -1.
template <bool BWD>
__global__ void __launch_bounds__(256)
tail_rows_kernel(const uint32_t* __restrict__ P, int M, int tiles, int W, int cap,
                 unsigned char* __restrict__ flags, int* __restrict__ row_slot,
                 int* __restrict__ row_drop, int* __restrict__ rows, RowState* __restrict__ state,
                 float* __restrict__ l0, int* __restrict__ dropped, int* __restrict__ n_over,
                 float inv_m) {
  __shared__ unsigned long long nnz_s;
  __shared__ int over_s, drop_s, warp_sum[8];
  __shared__ bool last_s;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid == 0) {
    nnz_s = 0;
    over_s = drop_s = 0;
  }
  __syncthreads();
  const size_t rw = (size_t)tiles * W;
  if (BWD) {
    const int r = blockIdx.x * 256 + tid;
    const bool f = r < M && (int)P[(size_t)r * rw] < 0;
    if (r < M) {
      flags[r] = f;
      row_slot[r] = -1;
    }
    const int n = __syncthreads_count(f);
    if (tid == 0) over_s = n;
  } else {
    for (int i = 0; i < 4; ++i) {
      const int r = blockIdx.x * 32 + warp * 4 + i;
      if (r >= M) break;
      int nnz = 0, drop = 0;
      for (int t = lane; t < tiles; t += 32) {
        const int c = (int)P[(size_t)r * rw + (size_t)t * W];
        nnz += c;
        drop += max(c - (W - 1), 0);
      }
      nnz = __reduce_add_sync(0xffffffffu, nnz);
      drop = __reduce_add_sync(0xffffffffu, drop);
      if (lane == 0) {
        flags[r] = drop > 0;
        row_slot[r] = -1;
        row_drop[r] = drop;
        atomicAdd(&nnz_s, (unsigned long long)nnz);
        if (drop > 0) {
          atomicAdd(&over_s, 1);
          atomicAdd(&drop_s, drop);
        }
      }
    }
  }
  __threadfence();
  __syncthreads();
  if (tid == 0) {
    if (!BWD) atomicAdd(&state->nnz, nnz_s);
    if (over_s != 0) atomicAdd(&state->n_over, over_s);
    if (!BWD && drop_s != 0) atomicAdd(&state->dropped, drop_s);
    __threadfence();
    last_s = atomicAdd(&state->done, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last_s) return;
  __threadfence();
  const int over = *(volatile int*)&state->n_over;
  int lost = *(volatile int*)&state->dropped;
  if (over > 0 && cap > 0) {
    const int per = (M + 255) / 256, r0 = tid * per, r1 = min(M, r0 + per);
    int mine = 0;
    for (int r = r0; r < r1; ++r) mine += __ldcg(flags + r);
    int inc = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += v;
    }
    if (lane == 31) warp_sum[warp] = inc;
    if (tid == 0) drop_s = 0;
    __syncthreads();
    int pos = inc - mine;
    for (int w = 0; w < warp; ++w) pos += warp_sum[w];
    int kept = 0;
    for (int r = r0; r < r1 && pos < cap; ++r) {
      if (!__ldcg(flags + r)) continue;
      rows[pos] = r;
      row_slot[r] = pos++;
      if (!BWD) kept += __ldcg(row_drop + r);
    }
    if (kept) atomicAdd(&drop_s, kept);
    __syncthreads();
    lost -= drop_s;
  }
  if (tid == 0) {
    state->n_tail = min(over, cap);
    if (!BWD) {
      *l0 = (float)(*(volatile unsigned long long*)&state->nnz) * inv_m;
      *dropped = lost;
      *n_over = over;
    }
  }
}

// One block per listed row: copies the row of x and (FLAG) sets the sign bit of its count words.
template <bool FLAG>
__global__ void __launch_bounds__(128)
tail_gather_kernel(uint32_t* __restrict__ P, const uint4* __restrict__ x,
                   const int* __restrict__ rows, const RowState* __restrict__ state,
                   uint4* __restrict__ xt, int tiles, int W, int vec_per_row) {
  if ((int)blockIdx.x >= state->n_tail) return;
  const int r = rows[blockIdx.x];
  if (FLAG)
    for (int t = threadIdx.x; t < tiles; t += 128)
      P[((size_t)r * tiles + t) * W] |= 0x80000000u;
  for (int v = threadIdx.x; v < vec_per_row; v += 128)
    xt[(size_t)blockIdx.x * vec_per_row + v] = __ldg(x + (size_t)r * vec_per_row + v);
}

// l1 = inv_m * sum of n partial sums, in a fixed order.
__global__ void __launch_bounds__(1024)
l1_sum_kernel(const float* __restrict__ part, int64_t n, float inv_m, float* __restrict__ l1) {
  __shared__ float warp_s[32];
  float s = 0.f;
  for (int64_t i = threadIdx.x; i < n; i += 1024) s += part[i];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) warp_s[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x < 32) {
    s = warp_s[threadIdx.x];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (threadIdx.x == 0) *l1 = s * inv_m;
  }
}

// Scratch of a training call; `tail` rows at most leave the slabs.  The [M, H] matrices are held for
// one chunk of rows; the weight gradients of several chunks add up in fp32 (carry).
struct TrainWs {
  RowState* state;
  unsigned char* flags;
  int *row_slot, *row_drop, *rows;
  __nv_bfloat16 *xt, *pt, *rt;   // tail rows: x, gate values, up products
  __nv_bfloat16 *t, *dru;        // [chunk, H] and (backward) [chunk, 2 H]
  float *l1_part, *part, *carry;
  int64_t chunk;
  size_t part_bytes, total;
};

TrainWs train_ws(void* base, int64_t M, int64_t D, int64_t H, int64_t tail, bool bwd,
                 int64_t max_rows) {
  unsigned char* p = static_cast<unsigned char*>(base);
  size_t off = 0;
  auto take = [&](size_t bytes) {
    unsigned char* q = p + off;
    off += align256(bytes);
    return q;
  };
  TrainWs w = {};
  w.chunk = chunk_rows(M, H, 1, max_rows);
  w.state = reinterpret_cast<RowState*>(take(sizeof(RowState)));
  w.flags = take((size_t)M);
  w.row_slot = reinterpret_cast<int*>(take((size_t)M * 4));
  w.row_drop = reinterpret_cast<int*>(take((size_t)M * 4));
  w.rows = reinterpret_cast<int*>(take((size_t)tail * 4));
  w.xt = reinterpret_cast<__nv_bfloat16*>(take((size_t)tail * D * 2));
  w.pt = reinterpret_cast<__nv_bfloat16*>(take((size_t)tail * H * 2));
  if (bwd) w.rt = reinterpret_cast<__nv_bfloat16*>(take((size_t)tail * H * 2));
  w.t = reinterpret_cast<__nv_bfloat16*>(take((size_t)w.chunk * H * 2));
  if (bwd) w.dru = reinterpret_cast<__nv_bfloat16*>(take((size_t)w.chunk * H * 4));
  const int64_t nt = H / pg::kTile, slots = sm_count() / 2;
  auto row_tiles = [](int64_t rows) { return (rows + pg::kTile - 1) / pg::kTile; };
  if (!bwd) w.l1_part = reinterpret_cast<float*>(take((size_t)row_tiles(M) * nt * 16 * 4));
  size_t part = 0;
  auto more = [&](size_t b) { part = b > part ? b : part; };
  if (!bwd) more(pg::part_bytes(row_tiles(M) * nt, (int)(D / kStageK), slots, false));
  const int64_t sizes[2] = {w.chunk, w.chunk > 0 ? M % w.chunk : 0};
  for (int64_t rows : sizes) {  // which tiles are cut depends on their number
    if (rows <= 0) continue;
    more(pg::part_bytes(row_tiles(rows) * nt, (int)(D / kStageK), slots, false));
    more(pg::part_bytes(row_tiles(rows) * (D / pg::kTile), (int)((bwd ? 2 : 1) * H / kStageK), slots,
                        true));
    if (bwd)
      more(pg::part_bytes(3 * nt * (D / pg::kTile), (int)((rows + kStageK - 1) / kStageK), slots,
                          false));
  }
  w.part = reinterpret_cast<float*>(take(part));
  w.part_bytes = part;
  if (bwd && w.chunk < M) w.carry = reinterpret_cast<float*>(take((size_t)3 * H * D * 4));
  w.total = off;
  return w;
}

// Dense products of the listed tail rows: out[i, :] = xt[i, :] w^T (relu), device-side row count.
int tail_product(const TrainWs& w, const void* weight, __nv_bfloat16* out, bool relu, int64_t tail,
                 int64_t D, int64_t H, cudaStream_t stream) {
  pg::Args a = base_args(tail, H, D);
  a.rows_ptr = &w.state->n_tail;
  a.out = out;
  a.ld = H;
  a.wide = 1;
  a.relu = relu;
  const pg::Operand ox = {w.xt, tail, D}, ow = {weight, H, D};
  return pg::launch<pg::kStore, false, false>("tail rows", ox, ox, ow, ow, a, tail, sm_count(),
                                              stream);
}

int train_check(const char* fn, int64_t M, int64_t D, int64_t H, int cf, int64_t tail,
                std::initializer_list<const void*> ptrs, const void* scratch) {
  if (int rc = check_dims(fn, M, D, H, cf)) return rc;
  if (M == 0) return fail(B200_EINVAL, "%s: M must be > 0", fn);
  if (tail < 0 || tail > M) return fail(B200_EINVAL, "%s: need 0 <= tail_rows <= M", fn);
  for (const void* p : ptrs) {
    if (p == nullptr) return fail(B200_ENULL, "%s: NULL pointer", fn);
    if (!aligned16(p)) return fail(B200_EALIGN, "%s: a pointer is not 16-byte aligned", fn);
  }
  if (scratch == nullptr) return fail(B200_ENULL, "%s: scratch is NULL", fn);
  if (reinterpret_cast<uintptr_t>(scratch) & 255u)
    return fail(B200_EALIGN, "%s: scratch is not 256-byte aligned", fn);
  return B200_OK;
}

// Device times of the parts of a call, added to ms[]; ms == nullptr: nothing is recorded.  Every part
// is waited for.
class Parts {
 public:
  Parts(float* ms, cudaStream_t stream) : ms_(ms), stream_(stream) {
    if (ms_ == nullptr) return;
    for (cudaEvent_t& e : event_) ok_ = cudaEventCreate(&e) == cudaSuccess && ok_;
    ok_ = ok_ && cudaEventRecord(event_[0], stream_) == cudaSuccess;
  }
  ~Parts() {
    for (cudaEvent_t e : event_)
      if (e != nullptr) cudaEventDestroy(e);
  }
  // Ends part `i`; the next one begins.
  void end(int i) {
    if (ms_ == nullptr || !ok_) return;
    float t = 0.f;
    ok_ = cudaEventRecord(event_[1], stream_) == cudaSuccess &&
          cudaEventSynchronize(event_[1]) == cudaSuccess &&
          cudaEventElapsedTime(&t, event_[0], event_[1]) == cudaSuccess;
    if (!ok_) return;
    ms_[i] += t;
    cudaEvent_t e = event_[0];
    event_[0] = event_[1];
    event_[1] = e;
  }
  int status(const char* fn) const {
    return ok_ ? B200_OK : fail(B200_ECUDA, "%s: the parts of the call could not be timed", fn);
  }

 private:
  float* ms_;
  cudaStream_t stream_;
  cudaEvent_t event_[2] = {nullptr, nullptr};
  bool ok_ = true;
};

int train_room(const char* fn, size_t have, size_t need) {
  if (have < need)
    return fail(B200_EWORKSPACE, "%s: scratch holds %zu bytes, %zu needed", fn, have, need);
  return B200_OK;
}

}  // namespace

}  // namespace b200

using namespace b200;

extern "C" size_t b200_hybrid_train_scratch_bytes_chunked(int64_t M, int64_t D, int64_t H,
                                                          int64_t tail_rows, int backward,
                                                          int64_t max_rows) {
  if (M <= 0 || D < 256 || H < 256 || H > 65536 || D % 256 || H % 256 || tail_rows < 0) return 0;
  return train_ws(nullptr, M, D, H, tail_rows, backward != 0, max_rows).total;
}

extern "C" size_t b200_hybrid_train_scratch_bytes(int64_t M, int64_t D, int64_t H, int64_t tail_rows,
                                                  int backward) {
  return b200_hybrid_train_scratch_bytes_chunked(M, D, H, tail_rows, backward, 0);
}

extern "C" int b200_hybrid_train_forward_timed(
    const void* x, const void* g, const void* k, const void* v, void* out, void* p_slab,
    void* r_slab, void* t_slab, float* l0, float* l1, int* dropped, int* n_over, int64_t M,
    int64_t D, int64_t H, int cf, int64_t tail_rows, void* workspace, size_t workspace_bytes,
    void* scratch, size_t scratch_bytes, int64_t max_rows, float* part_ms, void* stream) {
  const char* fn = "b200_hybrid_train_forward";
  if (int rc = train_check(fn, M, D, H, cf, tail_rows, {x, g, k, v, out, p_slab, r_slab, t_slab},
                           scratch))
    return rc;
  const TrainWs w = train_ws(scratch, M, D, H, tail_rows, false, max_rows);
  if (int rc = train_room(fn, scratch_bytes, w.total)) return rc;
  if (l0 == nullptr || l1 == nullptr || dropped == nullptr || n_over == nullptr)
    return fail(B200_ENULL, "%s: NULL result pointer", fn);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const SplitRoom room = {w.part, w.part_bytes, split_counters(workspace, workspace_bytes)};
  const int tiles = (int)(H / kTileN), W = kTileN / cf;
  const float inv_m = 1.f / (float)M;
  Parts parts(part_ms, st);
  if (cudaMemsetAsync(w.state, 0, sizeof(RowState), st) != cudaSuccess)
    return fail(B200_ECUDA, "%s: cudaMemsetAsync failed", fn);
  // the gate pattern
  pdl_suppressed() = true;  // its predecessor is the memset
  int rc = M > 128 && !tile_pack_serves(M, H)
               ? pair_pack(x, g, nullptr, p_slab, nullptr, M, D, H, cf, nullptr, room, st)
               : b200_twell_pack(x, g, nullptr, p_slab, M, D, H, cf, stream);
  pdl_suppressed() = false;
  if (rc) return rc;
  parts.end(0);
  tail_rows_kernel<false><<<(unsigned)((M + 31) / 32), 256, 0, st>>>(
      static_cast<const uint32_t*>(p_slab), (int)M, tiles, W, (int)tail_rows, w.flags, w.row_slot,
      w.row_drop, w.rows, w.state, l0, dropped, n_over, inv_m);
  if (int e = check_launch(fn)) return e;
  if (tail_rows > 0) {
    tail_gather_kernel<true><<<(unsigned)tail_rows, 128, 0, st>>>(
        static_cast<uint32_t*>(p_slab), static_cast<const uint4*>(x), w.rows, w.state,
        reinterpret_cast<uint4*>(w.xt), tiles, W, (int)(D / 8));
    if (int e = check_launch(fn)) return e;
    if (int e = tail_product(w, g, w.pt, true, tail_rows, D, H, st)) return e;
  }
  parts.end(1);
  // R, T and T v, chunk by chunk
  for (int64_t r0 = 0; r0 < M; r0 += w.chunk) {
    const int64_t m = M - r0 < w.chunk ? M - r0 : w.chunk;
    const void* xc = static_cast<const __nv_bfloat16*>(x) + r0 * D;
    pg::Args a = base_args(m, H, D);
    a.slab_w = W;
    a.row_words = tiles * W;
    a.slab_p = static_cast<uint32_t*>(p_slab) + r0 * a.row_words;
    a.slab_r = static_cast<uint32_t*>(r_slab) + r0 * a.row_words;
    a.slab_t = static_cast<uint32_t*>(t_slab) + r0 * a.row_words;
    a.row_slot = tail_rows > 0 ? w.row_slot + r0 : nullptr;
    a.tail_p = w.pt;
    a.l1_part = w.l1_part + r0 / pg::kTile * tiles * 16;  // chunks are whole row tiles
    pg::give_room(a, room);
    const pg::Operand ox = {xc, m, D}, ok = {k, H, D}, ot = {w.t, m, H};
    if (int e = pg::launch<pg::kFwd, false, false>(fn, ox, ot, ok, ot, a, m, sm_count(), st)) return e;
    parts.end(2);
    if (int e = pair_down(w.t, 1, v, static_cast<__nv_bfloat16*>(out) + r0 * D, m, D, H,
                          {nullptr, 0u, 0, nullptr}, room, st))
      return e;
    parts.end(3);
  }
  l1_sum_kernel<<<1, 1024, 0, st>>>(w.l1_part, (M + pg::kTile - 1) / pg::kTile * tiles * 16, inv_m,
                                    l1);
  parts.end(3);
  if (int e = parts.status(fn)) return e;
  return check_launch(fn);
}

extern "C" int b200_hybrid_train_forward_chunked(
    const void* x, const void* g, const void* k, const void* v, void* out, void* p_slab,
    void* r_slab, void* t_slab, float* l0, float* l1, int* dropped, int* n_over, int64_t M,
    int64_t D, int64_t H, int cf, int64_t tail_rows, void* workspace, size_t workspace_bytes,
    void* scratch, size_t scratch_bytes, int64_t max_rows, void* stream) {
  return b200_hybrid_train_forward_timed(x, g, k, v, out, p_slab, r_slab, t_slab, l0, l1, dropped,
                                         n_over, M, D, H, cf, tail_rows, workspace, workspace_bytes,
                                         scratch, scratch_bytes, max_rows, nullptr, stream);
}

extern "C" int b200_hybrid_train_forward(const void* x, const void* g, const void* k, const void* v,
                                         void* out, void* p_slab, void* r_slab, void* t_slab,
                                         float* l0, float* l1, int* dropped, int* n_over, int64_t M,
                                         int64_t D, int64_t H, int cf, int64_t tail_rows,
                                         void* workspace, size_t workspace_bytes, void* scratch,
                                         size_t scratch_bytes, void* stream) {
  return b200_hybrid_train_forward_chunked(x, g, k, v, out, p_slab, r_slab, t_slab, l0, l1, dropped,
                                           n_over, M, D, H, cf, tail_rows, workspace,
                                           workspace_bytes, scratch, scratch_bytes, 0, stream);
}

extern "C" int b200_hybrid_train_backward_timed(
    const void* x, const void* g, const void* k, const void* v, const void* p_slab,
    const void* r_slab, const void* g_out, const float* l1_grad, void* dx, void* dg, void* dk,
    void* dv, int64_t M, int64_t D, int64_t H, int cf, int64_t tail_rows, void* workspace,
    size_t workspace_bytes, void* scratch, size_t scratch_bytes, int64_t max_rows, float* part_ms,
    void* stream) {
  const char* fn = "b200_hybrid_train_backward";
  if (int rc = train_check(fn, M, D, H, cf, tail_rows,
                           {x, g, k, v, p_slab, r_slab, g_out, dx, dg, dk, dv}, scratch))
    return rc;
  const TrainWs w = train_ws(scratch, M, D, H, tail_rows, true, max_rows);
  if (int rc = train_room(fn, scratch_bytes, w.total)) return rc;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const SplitRoom room = {w.part, w.part_bytes, split_counters(workspace, workspace_bytes)};
  const int tiles = (int)(H / kTileN), W = kTileN / cf;
  Parts parts(part_ms, st);
  if (tail_rows > 0) {
    if (cudaMemsetAsync(w.state, 0, sizeof(RowState), st) != cudaSuccess)
      return fail(B200_ECUDA, "%s: cudaMemsetAsync failed", fn);
    tail_rows_kernel<true><<<(unsigned)((M + 255) / 256), 256, 0, st>>>(
        static_cast<const uint32_t*>(p_slab), (int)M, tiles, W, (int)tail_rows, w.flags, w.row_slot,
        w.row_drop, w.rows, w.state, nullptr, nullptr, nullptr, 0.f);
    tail_gather_kernel<false><<<(unsigned)tail_rows, 128, 0, st>>>(
        nullptr, static_cast<const uint4*>(x), w.rows, w.state, reinterpret_cast<uint4*>(w.xt),
        tiles, W, (int)(D / 8));
    if (int e = check_launch(fn)) return e;
    if (int e = tail_product(w, g, w.pt, true, tail_rows, D, H, st)) return e;
    if (int e = tail_product(w, k, w.rt, false, tail_rows, D, H, st)) return e;
    parts.end(0);
  }
  for (int64_t r0 = 0; r0 < M; r0 += w.chunk) {
    const int64_t m = M - r0 < w.chunk ? M - r0 : w.chunk;
    const void* xc = static_cast<const __nv_bfloat16*>(x) + r0 * D;
    const void* gc = static_cast<const __nv_bfloat16*>(g_out) + r0 * D;
    void* dxc = static_cast<__nv_bfloat16*>(dx) + r0 * D;
    // dT = g_out V^T on the pattern; dR = dT P, dU = dT R, T = R P
    pg::Args a = base_args(m, H, D);
    a.slab_w = W;
    a.row_words = tiles * W;
    a.slab_p = const_cast<uint32_t*>(static_cast<const uint32_t*>(p_slab)) + r0 * a.row_words;
    a.slab_r = const_cast<uint32_t*>(static_cast<const uint32_t*>(r_slab)) + r0 * a.row_words;
    a.row_slot = tail_rows > 0 ? w.row_slot + r0 : nullptr;
    a.tail_p = w.pt;
    a.tail_r = w.rt;
    a.l1_grad = l1_grad;
    a.inv_m = 1.f / (float)M;
    pg::give_room(a, room);
    const pg::Operand og = {gc, m, D}, ov = {v, H, D}, odu = {w.dru, m, 2 * H}, ot = {w.t, m, H};
    if (int e = pg::launch<pg::kBwd, false, false>(fn, og, odu, ov, ot, a, m, sm_count(), st)) return e;
    parts.end(1);
    // dX = [dR | dU] [K; G]
    pg::Args b = base_args(m, D, 2 * H);
    b.seg_ksteps = (int)(H / kStageK);
    b.out = static_cast<__nv_bfloat16*>(dxc);
    b.ld = D;
    b.wide = aligned32(dxc);
    pg::give_room(b, room);
    const pg::Operand odru = {w.dru, m, 2 * H}, okd = {k, D, H}, ogd = {g, D, H};
    if (int e = pg::launch<pg::kStore, false, true>(fn, odru, odru, okd, ogd, b, m, sm_count(), st))
      return e;
    parts.end(2);
    // [dK; dG] = [dR | dU]^T X and dV = T^T g_out in one launch
    pg::Args c = base_args(3 * H, D, m);
    c.second_mt = (int)(2 * H / pg::kTile);
    c.out = static_cast<__nv_bfloat16*>(dk);
    c.out_more[0] = static_cast<__nv_bfloat16*>(dg);
    c.out_more[1] = static_cast<__nv_bfloat16*>(dv);
    c.out_mt = (int)(H / pg::kTile);
    c.ld = D;
    c.wide = aligned32(dk) && aligned32(dg) && aligned32(dv);
    c.carry = w.carry;
    c.carry_in = r0 > 0;
    c.carry_out = r0 + m < M;
    pg::give_room(c, room);
    const pg::Operand a0 = {w.dru, 2 * H, m}, a1 = {w.t, H, m}, b0 = {xc, D, m}, b1 = {gc, D, m};
    const int e = w.carry == nullptr
                      ? pg::launch<pg::kStore, true, true>(fn, a0, a1, b0, b1, c, 3 * H, sm_count(), st)
                      : pg::launch<pg::kStoreCarry, true, true>(fn, a0, a1, b0, b1, c, 3 * H,
                                                                sm_count(), st);
    if (e) return e;
    parts.end(3);
  }
  return parts.status(fn);
}

extern "C" int b200_hybrid_train_backward_chunked(
    const void* x, const void* g, const void* k, const void* v, const void* p_slab,
    const void* r_slab, const void* g_out, const float* l1_grad, void* dx, void* dg, void* dk,
    void* dv, int64_t M, int64_t D, int64_t H, int cf, int64_t tail_rows, void* workspace,
    size_t workspace_bytes, void* scratch, size_t scratch_bytes, int64_t max_rows, void* stream) {
  return b200_hybrid_train_backward_timed(x, g, k, v, p_slab, r_slab, g_out, l1_grad, dx, dg, dk, dv,
                                          M, D, H, cf, tail_rows, workspace, workspace_bytes,
                                          scratch, scratch_bytes, max_rows, nullptr, stream);
}

extern "C" int b200_hybrid_train_backward(const void* x, const void* g, const void* k, const void* v,
                                          const void* p_slab, const void* r_slab,
                                          const void* g_out, const float* l1_grad, void* dx,
                                          void* dg, void* dk, void* dv, int64_t M, int64_t D,
                                          int64_t H, int cf, int64_t tail_rows, void* workspace,
                                          size_t workspace_bytes, void* scratch,
                                          size_t scratch_bytes, void* stream) {
  return b200_hybrid_train_backward_chunked(x, g, k, v, p_slab, r_slab, g_out, l1_grad, dx, dg, dk,
                                            dv, M, D, H, cf, tail_rows, workspace, workspace_bytes,
                                            scratch, scratch_bytes, 0, stream);
}

namespace b200 {

// Error word raised by a bounded wait that gave up (0 = none).  Reads and clears it; synchronises.
int pair_gemm_status() {
  int v = 0, zero = 0;
  if (cudaMemcpyFromSymbol(&v, pg::g_error, sizeof(int)) != cudaSuccess) return -1;
  if (v != 0) cudaMemcpyToSymbol(pg::g_error, &zero, sizeof(int));
  return v;
}

}  // namespace b200
