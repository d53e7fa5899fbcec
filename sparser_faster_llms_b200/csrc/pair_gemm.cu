// The fused MLPs on the paired tensor-core GEMM (pair_gemm.cuh) for calls of more than a few
// dozen tokens: gate GEMM with the pack epilogue, up GEMM whose epilogue multiplies by the slab
// pattern, down GEMM over the resulting hidden matrix.
#include "pair_gemm.cuh"

namespace b200 {

int sm_count();
int twell_t2d_launch(bool gated, bool hp, const void* x, const void* packed, const void* up,
                     const void* down, void* out, int64_t M, int64_t D, int64_t H, int cf,
                     void* workspace, size_t workspace_bytes, int sm_count, cudaStream_t stream,
                     const unsigned char* skip_rows, const FusedAr* fused_ar, const RunIf& run_if);

namespace {

constexpr int64_t kHiddenBytes = (int64_t)1 << 30;  // hidden matrix of one row chunk

int64_t chunk_rows(int64_t M, int64_t H, int terms) {
  const int64_t most = kHiddenBytes / (H * 2 * terms) / pg::kTile * pg::kTile;
  return M < most ? M : most;
}

size_t align256(size_t v) { return (v + 255) & ~(size_t)255; }

// Largest split-tile buffer of the three products of a chunk of `rows` rows.
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

}  // namespace

// Slabs of relu(x W^T + bias); `dense`: also the stored values as an [M, H] matrix.  part /
// counters may be null (no split of the last wave); entries: counter of stored entries or null.
int pair_pack(const void* x, const void* w, const float* bias, void* packed, void* dense, int64_t M,
              int64_t D, int64_t H, int cf, unsigned int* entries, float* part,
              unsigned int* counters, cudaStream_t stream) {
  pg::Args a = base_args(M, H, D);
  a.bias = bias;
  a.bias16 = aligned16(bias);
  a.entries = entries;
  a.slab_p = static_cast<uint32_t*>(packed);
  a.slab_w = kTileN / cf;
  a.row_words = (int)(H / kTileN) * a.slab_w;
  a.part = part;
  a.counters = counters;
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

// hidden[M, H] (hp: [M, 3 H]) = gate values of the slabs times x up^T on their pattern.
// row_slot / tail_p: rows whose gate values come from a dense matrix instead (may be null).
int pair_up(bool hp, const void* x, const void* packed, const void* up, void* hidden, int64_t M,
            int64_t D, int64_t H, int cf, const int* row_slot, const void* tail_p,
            const RunIf& run_if, float* part, unsigned int* counters, cudaStream_t stream) {
  pg::Args a = base_args(M, H, D);
  a.run_if = run_if;
  a.slab_p = const_cast<uint32_t*>(static_cast<const uint32_t*>(packed));
  a.slab_w = kTileN / cf;
  a.row_words = (int)(H / kTileN) * a.slab_w;
  a.row_slot = row_slot;
  a.tail_p = static_cast<const __nv_bfloat16*>(tail_p);
  a.out = static_cast<__nv_bfloat16*>(hidden);
  a.ld = hp ? 3 * H : H;
  a.wide = aligned32(hidden);
  a.part = part;
  a.counters = counters;
  const pg::Operand ox = {x, M, D}, ou = {up, H, D};
  return hp ? pg::launch<pg::kMulHp, false, false>("up product", ox, ox, ou, ou, a, M, sm_count(),
                                                   stream)
            : pg::launch<pg::kMul, false, false>("up product", ox, ox, ou, ou, a, M, sm_count(),
                                                 stream);
}

// out[M, D] = hidden[M, terms * H] [down; down; ...] with down [H, D] as it is stored.
int pair_down(const void* hidden, int terms, const void* down, void* out, int64_t M, int64_t D,
              int64_t H, const RunIf& run_if, float* part, unsigned int* counters,
              cudaStream_t stream) {
  pg::Args a = base_args(M, D, terms * H);
  a.run_if = run_if;
  a.seg_ksteps = (int)(H / kStageK);
  a.out = static_cast<__nv_bfloat16*>(out);
  a.ld = D;
  a.wide = aligned32(out);
  a.part = part;
  a.counters = counters;
  const pg::Operand oh = {hidden, M, terms * H}, od = {down, D, H};
  return pg::launch<pg::kStore, false, true>("down product", oh, oh, od, od, a, M, sm_count(),
                                             stream);
}

// Slabs and hidden matrix in one launch: the gate and up products of a tile follow one another in
// the two accumulators, and the pack epilogue of the first runs under the MMAs of the second.
// keep_all: hidden values are computed from every gate positive, not only from the stored ones.
int pair_gate_up(bool hp, const void* x, const void* gate, const float* bias, const void* up,
                 void* packed, void* hidden, int64_t M, int64_t D, int64_t H, int cf,
                 bool keep_all, cudaStream_t stream) {
  pg::Args a = base_args(M, H, D);
  a.bias = bias;
  a.bias16 = aligned16(bias);
  a.keep_all = keep_all;
  a.slab_p = static_cast<uint32_t*>(packed);
  a.slab_w = kTileN / cf;
  a.row_words = (int)(H / kTileN) * a.slab_w;
  a.out = static_cast<__nv_bfloat16*>(hidden);
  a.ld = hp ? 3 * H : H;
  a.wide = aligned32(hidden);
  const pg::Operand ox = {x, M, D}, og = {gate, H, D}, ou = {up, H, D};
  return hp ? pg::launch<pg::kGateUpHp, false, false>("gate and up products", ox, ox, og, ou, a, M,
                                                      sm_count(), stream)
            : pg::launch<pg::kGateUp, false, false>("gate and up products", ox, ox, og, ou, a, M,
                                                    sm_count(), stream);
}

namespace {

// Up and down rows together stay in L2, where a gathered entry is cheaper.
bool rows_in_l2(int64_t D, int64_t H) { return 4 * H * D <= (int64_t)100 << 20; }

// From this many tokens on the products are dense.  Measured under graph replay with weights from
// HBM, us per layer, gather form at 0.5 % / 2 % density -> dense form (any density):
//   D 1024, H 4096:   256 tokens 27 / 37 -> 34;  512 tokens 35 / 53 -> 35;  1024 tokens 41 / 73 -> 39
//   D 2048, H 8192:   128 tokens 32 / 48 -> 50;  256 tokens 48 / 84 -> 51;  512 tokens 69 / 140 -> 58
//   D 4096, H 16384:  64 tokens 91 (1 %) -> 93;  128 tokens 123 (1 %) -> 98
int64_t dense_from(int64_t D, int64_t H) {
  return D * H <= (int64_t)1 << 23 ? 320 : rows_in_l2(D, H) ? 160 : 96;
}

}  // namespace

// Which calls of the fused MLPs take this form.  High precision pays three down products, so it
// needs a larger call; the non-gated MLP saves only half as much.
bool pair_mlp_serves(int64_t M, int64_t D, int64_t H, bool gated, bool hp) {
  if (H < 2048) return false;  // few entries per token: nothing to gain
  if (hp) return M * D * H >= (int64_t)1 << 36;
  return M >= (gated ? 1 : 2) * dense_from(D, H);
}

// Whether the device chooses between the dense and the gather form of the up and down products by
// the stored entries of the call (two launches that return at once and a 4-byte memset, about
// 10 us); otherwise gate and up run in one launch and the dense form always.  At 0.5 % density
// the always-dense form is level with the gather form up to 4096 tokens (D 2048, H 8192: 305
// against 301 us) and ahead of it at D 1024 (88 against 96 us) and D 4096 (1152 against 1407 us).
// At 16384 tokens, D 2048, H 8192: gather 1070 us at 0.5 %, dense 1280 at any density, gather
// 2650 at 2 %.
static bool choose_on_device(int64_t M, int64_t D, int64_t H, bool gated, bool hp) {
  if (hp || !gated) return true;
  return M > 4096 && rows_in_l2(D, H) && 4 * H * D > (int64_t)32 << 20;
}

// Stored entries per token up to which the gather form is the faster one.  Measured (D 2048,
// H 8192): up + down 49 ns per token dense and 0.8 ns per entry gathered; high precision 104 ns;
// D 4096, H 16384 (rows from HBM as well): 176 ns against 2.7 ns, high precision 382 ns.
static int64_t gather_entries(int64_t D, int64_t H, bool hp) {
  return H * (hp ? 2 : 1) / (rows_in_l2(D, H) ? 128 : 224);
}

size_t pair_part_bytes(int64_t M, int64_t D, int64_t H) { return mlp_part_bytes(M, D, H, 1); }

size_t pair_mlp_scratch_bytes(int64_t M, int64_t D, int64_t H, bool gated, bool hp) {
  if (!pair_mlp_serves(M, D, H, gated, hp)) return 0;
  const int terms = hp ? 3 : 1;
  const int64_t rows = chunk_rows(M, H, terms);
  return align256((size_t)rows * H * 2 * terms) + 256 + mlp_part_bytes(rows, D, H, terms);
}

// workspace: the contraction workspace (its zero-filled counters; may be null).
int pair_mlp(bool gated, bool hp, const void* x, const void* gate, const float* bias,
             const void* up, const void* down, void* packed, void* out, int64_t M, int64_t D,
             int64_t H, int cf, void* workspace, size_t workspace_bytes, void* scratch,
             cudaStream_t stream) {
  const int terms = hp ? 3 : 1;
  const int64_t rows = chunk_rows(M, H, terms);
  const int64_t row_words = H / cf;
  unsigned char* p = static_cast<unsigned char*>(scratch) + align256((size_t)rows * H * 2 * terms);
  unsigned int* entries = reinterpret_cast<unsigned int*>(p);
  float* part = reinterpret_cast<float*>(p + 256);
  unsigned int* counters = workspace != nullptr && workspace_bytes >= 16384
                               ? static_cast<unsigned int*>(workspace)
                               : nullptr;
  for (int64_t r0 = 0; r0 < M; r0 += rows) {
    const int64_t m = M - r0 < rows ? M - r0 : rows;
    const void* xc = static_cast<const __nv_bfloat16*>(x) + r0 * D;
    void* pc = static_cast<uint32_t*>(packed) + r0 * row_words;
    void* oc = static_cast<__nv_bfloat16*>(out) + r0 * D;
    RunIf run_if = {nullptr, 0u};
    const bool choose = choose_on_device(m, D, H, gated, hp);
    if (choose) {
      const int64_t limit = m * gather_entries(D, H, hp);
      run_if = {entries, (unsigned int)(limit < 0x7fffffff ? limit : 0x7fffffff)};
      if (cudaMemsetAsync(entries, 0, sizeof(unsigned int), stream) != cudaSuccess)
        return fail(B200_ECUDA, "fused MLP: cudaMemsetAsync failed");
    }
    if (gated && !choose) {
      if (int rc = pair_gate_up(hp, xc, gate, bias, up, pc, scratch, m, D, H, cf, false, stream))
        return rc;
    } else {
      pdl_suppressed() = choose;  // its predecessor is the memset
      const int rc = pair_pack(xc, gate, bias, pc, gated ? nullptr : scratch, m, D, H, cf,
                               choose ? entries : nullptr, part, counters, stream);
      pdl_suppressed() = false;
      if (rc) return rc;
      if (gated)
        if (int rc = pair_up(hp, xc, pc, up, scratch, m, D, H, cf, nullptr, nullptr, run_if, part,
                             counters, stream))
          return rc;
    }
    if (int rc = pair_down(scratch, terms, down, oc, m, D, H, run_if, part, counters, stream))
      return rc;
    if (run_if.entries != nullptr)
      if (int rc = twell_t2d_launch(gated, hp, xc, pc, up, down, oc, m, D, H, cf, workspace,
                                    workspace_bytes, sm_count(), stream, nullptr, nullptr, run_if))
        return rc;
  }
  return B200_OK;
}

// Error word raised by a bounded wait that gave up (0 = none).  Reads and clears it; synchronises.
int pair_gemm_status() {
  int v = 0, zero = 0;
  if (cudaMemcpyFromSymbol(&v, pg::g_error, sizeof(int)) != cudaSuccess) return -1;
  if (v != 0) cudaMemcpyToSymbol(pg::g_error, &zero, sizeof(int));
  return v;
}

}  // namespace b200
