// Persistent tcgen05 GEMM on pairs of SMs (cta_group::2) with the sparse-FFN epilogues.
//
//   acc[m, n] = sum_k A[m, k] B[n, k]      bf16 operands, fp32 accumulators in TMEM
//
// A pair of CTAs (cluster of 2) computes 256 rows x 256 columns; CTA r holds rows
// [128 r, +128) of A, columns [128 r, +128) of B and the accumulator of its rows (TMEM lane =
// row, TMEM column = column).  A 64-k stage is 16 KB + 16 KB per CTA, i.e. 128 flop per staged
// byte: the rate of the 256 x 256 one-CTA tile, at half its TMEM, so that two accumulators fit and
// the epilogue of tile i runs under the MMAs of tile i + 1.
//
// Either operand may be K-major (rows of k-values) or MN-major (stored [k][m]): products with a
// transposed operand read the matrix where it lies, no transpose pass.  B can change after
// seg_ksteps k-steps (one accumulator over [A0 | A1] [B0; B1]) and both operands at row tile
// second_mt (several products in one launch).
//
// Work items: the first full_tiles tiles are one item each; each later tile (the last wave, or
// all tiles of a product too small to fill the GPU) is cut into `splits` ranges of k.  The warp
// that arrives last at a (tile, 32-row, column-half) block adds the ranges' fp32 sums in order
// and runs the epilogue on them, so the result does not depend on the arrival order.
//
// Roles per CTA (320 threads): warp 0 TMA producer, warp 1 MMA issuer (leader CTA only), warps
// 2..9 epilogue, two per TMEM lane quarter.  Barriers:
//   full[s]   leader:  both CTAs' copies of stage s have landed (the peer's copies signal it too)
//   empty[s]  each CTA: the MMAs have read stage s (multicast commit)
//   tfull[b]  each CTA: accumulator b is complete (multicast commit)
//   tempty[b] leader:  every epilogue warp of both CTAs has read accumulator b
// Every wait is bounded; a wait that gives up sets the error word, and the CTA pair leaves
// through the common cluster barrier, which frees TMEM.
#pragma once

#include <cooperative_groups.h>

#include "tc_common.cuh"

namespace b200 {
namespace {

namespace pg {

constexpr int kThreads = 320;
constexpr int kTile = 256;                   // rows and columns per pair
constexpr int kOperandBytes = 128 * 128;     // one CTA's half of A or B per 64-k stage
constexpr int kStageBytes = 2 * kOperandBytes;
constexpr int kBatch = 16;                   // slab rows whose words are in flight at a time
// k-steps per range of the up product in high precision; the ranges are added in fp32.  Error of the hidden
// values against 64 bits, N(0, 1) tokens: one range over D 2048 / 4096 2.1e-6 / 4.4e-6; ranges of 8 k-steps
// 4.8e-7, of 4 2.4e-7, of 1 1.3e-7 / 1.6e-7 (fp32 FMA chains 0.8e-7 / 0.9e-7).  y is off by 1.66e-3 with
// any of them.  A range costs the epilogue about 1.2 us: 777 tokens, D 2048, H 8192, 2 %, one range 110 us,
// of 8 k-steps 117, of 4 124, of 1 185; gathers 161.
constexpr int kDrain = 8;

enum Epilogue {
  kStore = 0,    // out[row, col] = bf16(acc)
  kPack = 1,     // TwELL slabs of relu(acc + bias)
  kPackDense = 6,  // the same, and the stored values as a dense matrix
  kGateUp = 7,   // kPack on a first accumulator (B0) and kMul with its values on a second (B1):
                 //   out = bf16(g * bf16(acc)) on the slab pattern, 0 elsewhere
  kGateUpHp = 8,  // kPack on B0, and its values times the sums on B1 in fp32, in the slots of the slab
  kMulHp = 3,    // g * acc in fp32, as three bf16 terms side by side (out row = [hi | mid | lo])
  kStoreCarry = 9,  // kStore on a product whose k comes in several launches: fp32 sums carried between
  kFwd = 4,      // training forward: R = bf16(acc) and T = R * P as slabs, T dense, l1 partial sums
  kBwd = 5       // training backward: dense [dR | dU] and T from acc = dT
};

// Shared memory of the eight epilogue warps: 32 rows x 256 bytes of pattern each, or the blocks of
// the training epilogues.
__host__ __device__ constexpr int buf_bytes(int epi) {
  return epi == kStore || epi == kStoreCarry ? 0 : epi == kBwd ? 8 * 3 * 4096 : 8 * 32 * 256;
}

struct Args {
  int rows;                  // rows of the product (device count in rows_ptr when not null)
  const int* rows_ptr;
  int n_tiles, ksteps, seg_ksteps, second_mt, group;
  int full_tiles, splits;    // see above; splits == 1: no split (full_tiles unused)
  float* sums;               // kStore, every tile split: fp32 sums [splits][rows][256 n_tiles]
  float* part;               // [items of split tiles][2][8 warps][128 columns][32 rows]
  unsigned int* counters;    // [split tiles][2][8], zero at rest
  size_t part_bytes;         // host: size of part
  __nv_bfloat16* out;        // dense result, row stride ld
  long long ld;
  int wide;                  // out rows are 32-byte aligned
  int relu;                  // kStore
  __nv_bfloat16* out_more[2];  // kStore: results of the row tiles from out_mt and 2 out_mt on
  int out_mt;                // 0: all rows in out
  float* carry;              // kStoreCarry: [tiles][2][8 warps][128 columns][32 rows] sums so far
  int carry_in, carry_out;   //   whether it is added, and whether it takes the sums instead of out
  const float* bias;         // packs; bias16: 16-byte aligned
  int bias16;
  // slab operands [rows][row_words], slab_w words per 256 columns
  uint32_t* slab_p;          // pattern and values (kPack: output)
  uint32_t* slab_r;          // kFwd: output, kBwd: input
  uint32_t* slab_t;          // kFwd: output
  int slab_w, row_words;
  // kFwd, kBwd, rows taken out of the slabs: row_slot[row] >= 0 is the row of tail_p / tail_r
  const int* row_slot;
  const __nv_bfloat16* tail_p;
  const __nv_bfloat16* tail_r;
  float* l1_part;            // kFwd: [tiles][16] sums of |T|
  const float* l1_grad;      // kBwd: device scalar or null
  float inv_m;
  float* values;             // kGateUpHp: [rows][row_words], hidden values of the stored entries
  int keep_all;              // kGateUp: values past a slab's capacity still count in the product
  unsigned int* entries;     // packs: stored entries are added here (may be null)
  RunIf run_if;
};

__device__ int g_error = 0;

__device__ __forceinline__ void tma_load(uint32_t dst, const CUtensorMap* map, int c0, int c1,
                                         uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes "
      "[%0], [%1, {%2, %3}], [%4];"
      ::"r"(dst), "l"(map), "r"(c0), "r"(c1), "r"(bar)
      : "memory");
}

__device__ __forceinline__ void mma(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc,
                                    uint32_t accumulate) {
  asm volatile(
      "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n}"
      ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(accumulate)
      : "memory");
}

// Arrives at the barrier of the same offset in both CTAs once all MMAs issued so far are done.
__device__ __forceinline__ void commit(uint64_t* bar) {
  asm volatile(
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 "
      "[%0], %1;"
      ::"r"(smem_u32(bar)), "h"((uint16_t)3)
      : "memory");
}

__device__ __forceinline__ void arrive_leader(uint64_t* bar) {
  asm volatile(
      "{\n.reg .b32 a;\nmapa.shared::cluster.u32 a, %0, 0;\n"
      "mbarrier.arrive.release.cluster.shared::cluster.b64 _, [a];\n}"
      ::"r"(smem_u32(bar))
      : "memory");
}

// MN-major operand, 128-byte swizzle: 64 x 64 boxes of 8 KB, 8-k groups 1024 B apart.
__device__ __forceinline__ uint64_t desc_mn(uint32_t saddr) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr & 0x3FFFFu) >> 4);
  d |= (uint64_t)(8192 >> 4) << 16;           // next 64 rows / columns
  d |= (uint64_t)(1024 >> 4) << 32;           // next 8 k
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)2 << 61;
  return d;
}

// Item t -> tile and range of k-steps; the split tile's index and the item's place in part[].
struct Item {
  int tile, k0, k1, split_tile, split;
};
__device__ __forceinline__ Item item_of(int t, const Args& a) {
  Item it = {t, 0, a.ksteps, -1, 0};
  if (a.splits > 1 && t >= a.full_tiles) {
    const int j = t - a.full_tiles;
    it.split_tile = j / a.splits;
    it.split = j - it.split_tile * a.splits;
    it.tile = a.full_tiles + it.split_tile;
    it.k0 = it.split * a.ksteps / a.splits;
    it.k1 = (it.split + 1) * a.ksteps / a.splits;
  }
  return it;
}

__device__ __forceinline__ void tile_of(int t, int m_tiles, const Args& a, int& mt, int& nt) {
  const int per = a.group * a.n_tiles;
  const int g = t / per, first = g * a.group, in = t - g * per;
  const int rows = min(a.group, m_tiles - first);
  mt = first + in % rows;
  nt = in / rows;
}

__device__ __forceinline__ uint32_t pack2(float a, float b) {
  __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&v);
}
__device__ __forceinline__ uint32_t mul2(uint32_t a, uint32_t b) {
  __nv_bfloat162 v = __hmul2(*reinterpret_cast<__nv_bfloat162*>(&a),
                             *reinterpret_cast<__nv_bfloat162*>(&b));
  return *reinterpret_cast<uint32_t*>(&v);
}
// 0xFFFF per half whose value is not +-0.
__device__ __forceinline__ uint32_t nonzero2(uint32_t a) {
  const __nv_bfloat162 z = __floats2bfloat162_rn(0.f, 0.f);
  return __hne2_mask(*reinterpret_cast<__nv_bfloat162*>(&a), z);
}
__device__ __forceinline__ float lo_f(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float hi_f(uint32_t w) { return __uint_as_float(w & 0xFFFF0000u); }

// 64 consecutive bytes (32 bf16) of one row per lane; `wide`: the row is 32-byte aligned, so a
// lane fills whole sectors with 256-bit stores.
__device__ __forceinline__ void store64(__nv_bfloat16* p, const uint32_t (&w)[16], int wide) {
  if (wide) {
#pragma unroll
    for (int i = 0; i < 2; ++i)
      asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
                   ::"l"(p + i * 16), "r"(w[8 * i]), "r"(w[8 * i + 1]), "r"(w[8 * i + 2]),
                     "r"(w[8 * i + 3]), "r"(w[8 * i + 4]), "r"(w[8 * i + 5]), "r"(w[8 * i + 6]),
                     "r"(w[8 * i + 7])
                   : "memory");
  } else {
#pragma unroll
    for (int i = 0; i < 4; ++i)
      reinterpret_cast<uint4*>(p)[i] = make_uint4(w[4 * i], w[4 * i + 1], w[4 * i + 2], w[4 * i + 3]);
  }
}

// Byte `off` of row `row` in a warp's pattern buffer: 256 bytes per row, 16-byte pieces swizzled so
// that 32 lanes reading the same piece of their own rows hit all banks.
__device__ __forceinline__ unsigned char* at(unsigned char* buf, int row, int off) {
  return buf + row * 256 + ((off & ~15) ^ ((row & 7) << 4)) + (off & 15);
}

// Pattern buffer of one warp: 32 rows x 128 columns of bf16 values (zero where nothing is stored),
// filled from the slabs of tile `nt`, columns [128 half, +128).
__device__ __forceinline__ void load_values(const Args& a, unsigned char* buf, int row0, int rows,
                                            int nt, int half, int lane) {
#pragma unroll
  for (int i = 0; i < 16; ++i)
    *reinterpret_cast<uint4*>(buf + lane * 256 + i * 16) = make_uint4(0u, 0u, 0u, 0u);
  __syncwarp();
  const uint32_t* base = a.slab_p + (size_t)nt * a.slab_w;
  for (int t0 = 0; t0 < 32; t0 += kBatch) {
    if (row0 + t0 >= rows) break;
    int cnt[kBatch], most = 0;
    for (int w0 = 0; w0 < a.slab_w; w0 += 32) {
      uint32_t w[kBatch];
#pragma unroll
      for (int j = 0; j < kBatch; ++j) {
        const int row = row0 + t0 + j;
        w[j] = row < rows ? base[(size_t)row * a.row_words + w0 + lane] : 0u;
      }
#pragma unroll
      for (int j = 0; j < kBatch; ++j) {
        if (w0 == 0) {
          cnt[j] = min(max((int)__shfl_sync(0xffffffffu, w[j], 0), 0), a.slab_w - 1);
          most = max(most, cnt[j]);
        }
        const int slot = w0 + lane, col = (int)(w[j] & 255u);
        if (slot >= 1 && slot <= cnt[j] && (col >> 7) == half)
          *reinterpret_cast<uint16_t*>(at(buf, t0 + j, (col & 127) * 2)) =
              (uint16_t)(w[j] >> 16);
      }
      if (most < w0 + 32) break;
    }
  }
  __syncwarp();
}

// The 32 sums of a lane's row in the 32 columns at `col` of the warp's block: from TMEM, or, for a
// split tile, the ranges' sums added in order.
struct Source {
  uint32_t acc;         // TMEM address of the block's first column
  const float* part;    // null: TMEM
  int splits;
};
constexpr size_t kItemFloats = (size_t)kTile * kTile;

__device__ __forceinline__ void fetch32(const Source& src, int cb, float (&v)[32]) {
  if (src.part == nullptr) {
    tmem_ld32(src.acc + (uint32_t)(cb * 32), v);
    return;
  }
#pragma unroll
  for (int c = 0; c < 32; ++c) v[c] = 0.f;
  for (int sp = 0; sp < src.splits; sp += 2) {  // two ranges in flight at a time
    const float* p = src.part + (size_t)sp * kItemFloats + cb * 1024;
    const bool two = sp + 1 < src.splits;
    float u[32], w[32];
#pragma unroll
    for (int c = 0; c < 32; ++c) {
      u[c] = __ldcg(p + c * 32);
      w[c] = two ? __ldcg(p + kItemFloats + c * 32) : 0.f;
    }
#pragma unroll
    for (int c = 0; c < 32; ++c) v[c] = (v[c] + u[c]) + w[c];
  }
}

// ---- training epilogues: sums -> slab entries and zero-filled dense tiles -----------------------
// Only 1 - 3 % of the sums are on the pattern, so the arithmetic runs per stored entry instead of
// per column: a 64-column block of sums goes to shared memory as bf16, the lanes pick their
// entries out of it, and the dense operands of the following products are zero-filled blocks with
// the entries scattered in, written by TMA (128-byte rows, clipped at the last row).  What bounds
// them is the dense writes and the MMAs of the next tile.  Against expanding the pattern to a dense
// tile and computing every column (two warps per scheduler, some 5000 instructions per warp and
// tile), 16384 tokens, D 1024, H 4096, 1 %: forward 229 -> 114 us, backward 317 -> 161 us (134 and
// 403 MB written: 22 and 67 us at copy speed; the product alone 96 us).  The backward gives up one
// of five operand stages for its third block per warp.

constexpr int kBlockBytes = 32 * 128;        // 32 rows x 64 columns of bf16, 128-byte swizzle
constexpr int kAhead = 16;                   // slab words per row that are fetched ahead

// Byte of column `col` in row `row` of a block: the layout of SWIZZLE_128B.
__device__ __forceinline__ unsigned char* blk(unsigned char* buf, int row, int col) {
  return buf + row * 128 + ((((col >> 3) ^ row) & 7) << 4) + (col & 7) * 2;
}
__device__ __forceinline__ void zero_row(unsigned char* buf, int row) {
#pragma unroll
  for (int i = 0; i < 8; ++i)
    *reinterpret_cast<uint4*>(buf + row * 128 + ((i ^ (row & 7)) << 4)) = make_uint4(0u, 0u, 0u, 0u);
}
__device__ __forceinline__ uint32_t lds16(const unsigned char* p) {
  return *reinterpret_cast<const uint16_t*>(p);
}
__device__ __forceinline__ void sts16(unsigned char* p, uint32_t v) {
  *reinterpret_cast<uint16_t*>(p) = (uint16_t)v;
}
__device__ __forceinline__ void tma_store(const CUtensorMap* map, const void* src, int c0, int c1) {
  asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%1, %2}], [%3];"
               ::"l"(map), "r"(c0), "r"(c1), "r"(smem_u32(src))
               : "memory");
}
__device__ __forceinline__ void tma_store_commit() {
  asm volatile("cp.async.bulk.commit_group;" ::: "memory");
}
__device__ __forceinline__ void tma_store_wait_read() {
  asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
}
__device__ __forceinline__ void tma_store_wait() {
  asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
}

// Slab words [w0, w0 + 16) of the warp's 32 rows: register pair g of a lane holds words
// w0 + 2 (lane & 7) and the next of row 4 g + lane / 8, i.e. 64 contiguous bytes per row.
__device__ __forceinline__ void load_words(const uint32_t* slab, const Args& a, int row0, int rows,
                                           int nt, int w0, int lane, uint2 (&w)[8]) {
  const size_t off = (size_t)nt * a.slab_w + w0 + (lane & 7) * 2;
#pragma unroll
  for (int g = 0; g < 8; ++g) {
    const int row = row0 + g * 4 + (lane >> 3);
    w[g] = row < rows ? *reinterpret_cast<const uint2*>(slab + (size_t)row * a.row_words + off)
                      : make_uint2(0u, 0u);
  }
}

// Stored entries per row (as load_words lays rows out) and the largest count of the 32 rows.
// Counts with the sign bit set belong to rows taken out of the slabs: no entries.
__device__ __forceinline__ int row_counts(const Args& a, const uint2 (&w)[8], int lane, int (&cnt)[8]) {
  int most = 0;
#pragma unroll
  for (int g = 0; g < 8; ++g) {
    cnt[g] = min(max((int)__shfl_sync(0xffffffffu, w[g].x, lane & 24), 0), a.slab_w - 1);
    most = max(most, cnt[g]);
  }
  return __reduce_max_sync(0xffffffffu, most);
}

// dT of one column pair (or one column in the low half): the bf16 sum, shifted by the l1 gradient
// times the sign of R.
__device__ __forceinline__ uint32_t shifted2(uint32_t dt, uint32_t r2, float shift) {
  if (shift == 0.f) return dt;
  const float r0 = lo_f(r2), r1 = hi_f(r2);
  const float s0 = r0 > 0.f ? shift : (r0 < 0.f ? -shift : 0.f);
  const float s1 = r1 > 0.f ? shift : (r1 < 0.f ? -shift : 0.f);
  return pack2(lo_f(dt) + s0, hi_f(dt) + s1);
}

// Sums of columns [64 hc, +64) of the warp's block as bf16 rows (lane = row).
__device__ __forceinline__ void sums_to_block(const Source& src, int hc, unsigned char* buf, int lane) {
#pragma unroll
  for (int cb = 0; cb < 2; ++cb) {
    float v[32];
    fetch32(src, hc * 2 + cb, v);
#pragma unroll
    for (int j = 0; j < 4; ++j)
      *reinterpret_cast<uint4*>(buf + lane * 128 + (((cb * 4 + j) ^ (lane & 7)) << 4)) =
          make_uint4(pack2(v[8 * j], v[8 * j + 1]), pack2(v[8 * j + 2], v[8 * j + 3]),
                     pack2(v[8 * j + 4], v[8 * j + 5]), pack2(v[8 * j + 6], v[8 * j + 7]));
  }
}

// Calls f(row, column in the 64-column block, slab offset, P word, R word) for this lane's stored
// entries of block `quarter` of tile nt; pw / rw hold the first kAhead words of every row.
template <bool WITH_R, typename F>
__device__ __forceinline__ void for_entries(const Args& a, int row0, int rows, int nt, int quarter,
                                            int lane, const uint2 (&pw)[8], const uint2 (&rw)[8],
                                            const int (&cnt)[8], int most, F f) {
  auto batch = [&](int w0, const uint2 (&p)[8], const uint2 (&r)[8]) {
#pragma unroll
    for (int g = 0; g < 8; ++g) {
      const int row = g * 4 + (lane >> 3), slot = w0 + (lane & 7) * 2;
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const uint32_t w = e == 0 ? p[g].x : p[g].y;
        if (slot + e >= 1 && slot + e <= cnt[g] && ((int)(w & 255u) >> 6) == quarter)
          f(row, (int)(w & 63u),
            (size_t)(row0 + row) * a.row_words + (size_t)nt * a.slab_w + slot + e, w,
            WITH_R ? (e == 0 ? r[g].x : r[g].y) : 0u);
      }
    }
  };
  batch(0, pw, rw);
#pragma unroll 1
  for (int w0 = kAhead; w0 <= most; w0 += kAhead) {
    uint2 p[8], r[8];
    load_words(a.slab_p, a, row0, rows, nt, w0, lane, p);
    if (WITH_R) load_words(a.slab_r, a, row0, rows, nt, w0, lane, r);
    batch(w0, p, r);
  }
}

// Calls f(row, offset of this lane's two columns in the rows of tail_p / tail_r, their place in the
// block) for every row of the warp that is out of the slabs; all lanes take part.
template <typename F>
__device__ __forceinline__ void for_tail_rows(const Args& a, int slot, int nt, int quarter, int lane,
                                              F f) {
  uint32_t todo = __ballot_sync(0xffffffffu, slot >= 0);
  while (todo != 0u) {
    const int t = __ffs(todo) - 1;
    todo &= todo - 1;
    const int s = __shfl_sync(0xffffffffu, slot, t);
    f(t, (size_t)s * a.n_tiles * kTile + nt * kTile + quarter * 64 + lane * 2, lane * 2);
  }
}

// Training forward: R and T in the slots of P, T as a dense matrix, this lane's part of sum |T|.
// buf: two blocks.  release() is called once the accumulator has been read.
template <typename Release>
__device__ __forceinline__ float forward_tile(const Args& a, const CUtensorMap* map_t, const Source& src,
                                              unsigned char* buf, int row0, int rows, int nt, int half,
                                              int lane, const uint2 (&pw)[8], int tail_slot,
                                              Release release) {
  int cnt[8];
  const int most = row_counts(a, pw, lane, cnt);
  unsigned char *bx = buf, *bt = buf + kBlockBytes;
  float l1 = 0.f;
  if (half == 0 && (lane & 7) == 0) {
#pragma unroll
    for (int g = 0; g < 8; ++g) {
      const int row = row0 + g * 4 + (lane >> 3);
      if (row >= rows) continue;
      const size_t off = (size_t)row * a.row_words + (size_t)nt * a.slab_w;
      a.slab_r[off] = pw[g].x;
      a.slab_t[off] = pw[g].x;
    }
  }
#pragma unroll 1
  for (int hc = 0; hc < 2; ++hc) {
    const int quarter = 2 * half + hc;
    if (lane == 0) tma_store_wait_read();
    __syncwarp();
    sums_to_block(src, hc, bx, lane);
    zero_row(bt, lane);
    if (hc == 1) release();
    __syncwarp();
    for_entries<false>(a, row0, rows, nt, quarter, lane, pw, pw, cnt, most,
                       [&](int row, int col, size_t off, uint32_t p, uint32_t) {
                         const uint32_t m = nonzero2(p >> 16);
                         const uint32_t r = lds16(blk(bx, row, col)) & m;
                         const uint32_t t = mul2(p >> 16, r) & m;
                         l1 += fabsf(lo_f(t));
                         sts16(blk(bt, row, col), t);
                         a.slab_r[off] = (p & 0xFFFFu) | (r << 16);
                         a.slab_t[off] = (p & 0xFFFFu) | (t << 16);
                       });
    for_tail_rows(a, tail_slot, nt, quarter, lane, [&](int row, size_t off, int col) {
      const uint32_t p2 = *reinterpret_cast<const uint32_t*>(a.tail_p + off), m = nonzero2(p2);
      const uint32_t r2 = *reinterpret_cast<const uint32_t*>(blk(bx, row, col)) & m;
      const uint32_t t2 = mul2(p2, r2) & m;
      l1 += fabsf(lo_f(t2));
      l1 += fabsf(hi_f(t2));
      *reinterpret_cast<uint32_t*>(blk(bt, row, col)) = t2;
    });
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncwarp();
    if (lane == 0 && row0 < rows) {
      tma_store(map_t, bt, nt * kTile + quarter * 64, row0);
      tma_store_commit();
    }
  }
  return l1;
}

// Training backward: dense [dR | dU] and T from dT.  buf: three blocks; the one that held dT is
// used again for T.
template <typename Release>
__device__ __forceinline__ void backward_tile(const Args& a, const CUtensorMap* map_dru,
                                              const CUtensorMap* map_t, const Source& src,
                                              unsigned char* buf, int row0, int rows, int nt, int half,
                                              int lane, const uint2 (&pw)[8], const uint2 (&rw)[8],
                                              int tail_slot, float shift, Release release) {
  int cnt[8];
  const int most = row_counts(a, pw, lane, cnt);
  unsigned char *bx = buf, *br = buf + kBlockBytes, *bu = buf + 2 * kBlockBytes;
#pragma unroll 1
  for (int hc = 0; hc < 2; ++hc) {
    const int quarter = 2 * half + hc;
    if (lane == 0) tma_store_wait_read();
    __syncwarp();
    sums_to_block(src, hc, bx, lane);
    zero_row(br, lane);
    zero_row(bu, lane);
    if (hc == 1) release();
    __syncwarp();
    for_entries<true>(a, row0, rows, nt, quarter, lane, pw, rw, cnt, most,
                      [&](int row, int col, size_t, uint32_t p, uint32_t r) {
                        p >>= 16;
                        r >>= 16;
                        const uint32_t m = nonzero2(p);
                        const uint32_t dt = shifted2(lds16(blk(bx, row, col)), r, shift) & m;
                        sts16(blk(br, row, col), mul2(dt, p) & m);
                        sts16(blk(bu, row, col), mul2(dt, r) & m);
                      });
    for_tail_rows(a, tail_slot, nt, quarter, lane, [&](int row, size_t off, int col) {
      const uint32_t p2 = *reinterpret_cast<const uint32_t*>(a.tail_p + off), m = nonzero2(p2);
      const uint32_t r2 = *reinterpret_cast<const uint32_t*>(a.tail_r + off);
      const uint32_t dt =
          shifted2(*reinterpret_cast<const uint32_t*>(blk(bx, row, col)), r2, shift) & m;
      *reinterpret_cast<uint32_t*>(blk(br, row, col)) = mul2(dt, p2) & m;
      *reinterpret_cast<uint32_t*>(blk(bu, row, col)) = mul2(dt, r2) & m;
    });
    __syncwarp();
    zero_row(bx, lane);
    __syncwarp();
    for_entries<true>(a, row0, rows, nt, quarter, lane, pw, rw, cnt, most,
                      [&](int row, int col, size_t, uint32_t p, uint32_t r) {
                        p >>= 16;
                        sts16(blk(bx, row, col), mul2(r >> 16, p) & nonzero2(p));
                      });
    for_tail_rows(a, tail_slot, nt, quarter, lane, [&](int row, size_t off, int col) {
      const uint32_t p2 = *reinterpret_cast<const uint32_t*>(a.tail_p + off);
      const uint32_t r2 = *reinterpret_cast<const uint32_t*>(a.tail_r + off);
      *reinterpret_cast<uint32_t*>(blk(bx, row, col)) = mul2(r2, p2) & nonzero2(p2);
    });
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncwarp();
    if (lane == 0 && row0 < rows) {
      const int c = nt * kTile + quarter * 64;
      tma_store(map_dru, br, c, row0);
      tma_store(map_dru, bu, a.n_tiles * kTile + c, row0);
      tma_store(map_t, bx, c, row0);
      tma_store_commit();
    }
  }
}

// First term of h where rounding h to bf16 would leave bf16's range, and what it leaves: infinities
// stand alone (inf - inf would put a NaN into the other terms), finite values keep the largest bf16.
constexpr float kBf16Max = 0x1.FEp127f;
__device__ __forceinline__ float first_term(float h) {
  return fabsf(h) > kBf16Max && !isinf(h) ? copysignf(kBf16Max, h) : h;
}
__device__ __forceinline__ float rest_of(float h, float first) { return isinf(h) ? 0.f : h - first; }

// h = g * u of 32 columns as three bf16 terms (24 bits of h), zero where g is.
__device__ __forceinline__ void mul_hp(const uint4* g4, const float (&v)[32], uint32_t (&w0)[16],
                                       uint32_t (&w1)[16], uint32_t (&w2)[16]) {
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const uint32_t g[4] = {g4[j].x, g4[j].y, g4[j].z, g4[j].w};
#pragma unroll
    for (int p = 0; p < 4; ++p) {
      const int c = 8 * j + 2 * p, o = 4 * j + p;
      const float g0 = lo_f(g[p]), g1 = hi_f(g[p]);
      float h0 = g0 != 0.f ? g0 * v[c] : 0.f, h1 = g1 != 0.f ? g1 * v[c + 1] : 0.f;
      w0[o] = pack2(h0, h1);
      if (fmaxf(fabsf(h0), fabsf(h1)) > kBf16Max) {
        w0[o] = pack2(first_term(h0), first_term(h1));
        h0 = rest_of(h0, lo_f(w0[o]));
        h1 = rest_of(h1, hi_f(w0[o]));
      } else {
        h0 -= lo_f(w0[o]);
        h1 -= hi_f(w0[o]);
      }
      w1[o] = pack2(h0, h1);
      h0 -= lo_f(w1[o]);
      h1 -= hi_f(w1[o]);
      w2[o] = pack2(h0, h1);
    }
  }
}

template <int EPI, bool A_MN, bool B_MN, int STAGES>
__global__ void __launch_bounds__(kThreads, 1)
pair_gemm_kernel(const __grid_constant__ CUtensorMap map_a0,
                 const __grid_constant__ CUtensorMap map_a1,
                 const __grid_constant__ CUtensorMap map_b0,
                 const __grid_constant__ CUtensorMap map_b1, const __grid_constant__ Args a) {
  constexpr uint32_t kIdesc = umma_idesc(256, 256) | (A_MN ? 1u << 15 : 0u) | (B_MN ? 1u << 16 : 0u);
  constexpr bool kGate2 = EPI == kGateUp || EPI == kGateUpHp;
  constexpr bool kIsPack = EPI == kPack || EPI == kPackDense || kGate2;
  constexpr bool kTrain = EPI == kFwd || EPI == kBwd;
  constexpr bool kPlain = EPI == kStore || EPI == kStoreCarry;
  constexpr int kBufBytes = buf_bytes(EPI) / 8;  // of one epilogue warp
  constexpr int kPhases = kGate2 ? 2 : 1;  // accumulators per item

  // Without a device-side choice or row count the set-up below runs while the predecessor drains.
  const bool early_wait = a.run_if.entries != nullptr || a.rows_ptr != nullptr;
  if (early_wait) pdl_wait();
  bool gate_only = false;  // kGateUp: the gather form follows, slabs are all that it needs
  if (a.run_if.entries != nullptr && !stored_more(a.run_if)) {
    if (EPI != kGateUp) return;
    gate_only = true;
  }
  const int phases = gate_only ? 1 : kPhases;
  const int rows = a.rows_ptr != nullptr ? *a.rows_ptr : a.rows;
  const int m_tiles = (rows + kTile - 1) / kTile;
  const int tiles = m_tiles * a.n_tiles;
  const int total = a.splits > 1 ? a.full_tiles + (tiles - a.full_tiles) * a.splits : tiles;
  const int pair = (int)blockIdx.x >> 1, pairs = (int)gridDim.x >> 1;
  if (pair >= total) return;  // the same for both CTAs: nothing allocated, no barrier used yet

  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>(
      (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  __shared__ __align__(8) uint64_t full_bar[STAGES], empty_bar[STAGES], tfull_bar[2], tempty_bar[2];
  __shared__ uint32_t tmem_slot;
  __shared__ volatile int abort_s;
  __shared__ int half_count[kIsPack ? 2 : 1][kIsPack ? 128 : 1];
  __shared__ volatile int last_s[4];

  cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
  const int crank = (int)blockIdx.x & 1;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
#pragma unroll
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
#pragma unroll
    for (int b = 0; b < 2; ++b) {
      mbar_init(&tfull_bar[b], 1);
      mbar_init(&tempty_bar[b], 16);
    }
    abort_s = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&map_a0) : "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&map_b0) : "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;"
                 ::"r"(smem_u32(&tmem_slot)), "r"(512)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  cluster.sync();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem_base = tmem_slot;
  if (!early_wait) pdl_wait();

  if (warp == 0) {
    // ---- TMA producer ----
    // The producer and the MMA thread bound the k-step (630 clocks against 512 of its MMAs when each step
    // computed its stage and descriptors in a lane == 0 branch): stage and phase are counted, descriptors
    // are a base plus an offset, and a wait that gives up ends the role.  4096 tokens, D 4096, H 16384
    // 1298 -> 1186 us; 2048 tokens, D 2048, H 8192 190 -> 172; training step of 16384 tokens 1138 -> 1045.
    if (elect_one()) {
      const uint32_t ring = smem_u32(smem);
      // both CTAs' copies are counted at the leader's barrier (bit 24 of a shared-window address is
      // the CTA's rank in the pair)
      const uint32_t leader_full = smem_u32(full_bar) & 0xFEFFFFFFu;
      int s = 0;
      uint32_t phase = 1;
      bool ok = true;
#pragma unroll 1
      for (int t = pair; t < total && ok; t += pairs) {
        const Item im = item_of(t, a);
        int mt, nt;
        tile_of(im.tile, m_tiles, a, mt, nt);
        const bool second = mt >= a.second_mt;
        const CUtensorMap* ma = second ? &map_a1 : &map_a0;
        const int ra = (second ? mt - a.second_mt : mt) * kTile + crank * 128;
        const int rb = nt * kTile + crank * 128;
#pragma unroll 1
        for (int ph = 0; ph < phases && ok; ++ph) {
          int kb = im.k0 % a.seg_ksteps;
          const CUtensorMap* mb =
              ph == 1 || second || im.k0 >= a.seg_ksteps ? &map_b1 : &map_b0;
#pragma unroll 1
          for (int k = im.k0; k < im.k1; ++k) {
            if (kb == a.seg_ksteps) {
              kb = 0;
              mb = &map_b1;
            }
            if (!mbar_wait(&empty_bar[s], phase)) {
              ok = false;
              break;
            }
            const uint32_t bar = leader_full + (uint32_t)s * 8u;
            if (crank == 0) mbar_expect_tx(&full_bar[s], 2 * kStageBytes);
            const uint32_t st = ring + (uint32_t)s * kStageBytes;
            if (A_MN) {
              tma_load(st, ma, ra, k * kStageK, bar);
              tma_load(st + 8192, ma, ra + 64, k * kStageK, bar);
            } else {
              tma_load(st, ma, k * kStageK, ra, bar);
            }
            if (B_MN) {
              tma_load(st + kOperandBytes, mb, rb, kb * kStageK, bar);
              tma_load(st + kOperandBytes + 8192, mb, rb + 64, kb * kStageK, bar);
            } else {
              tma_load(st + kOperandBytes, mb, kb * kStageK, rb, bar);
            }
            ++kb;
            if (++s == STAGES) {
              s = 0;
              phase ^= 1u;
            }
          }
        }
      }
      const int next = s;
      const uint32_t pass = phase;
      // the commits of the last stages must have arrived before this CTA may leave
#pragma unroll 1
      for (int i = 0; i < STAGES && ok; ++i) {
        ok = mbar_wait(&empty_bar[s], phase);
        if (++s == STAGES) {
          s = 0;
          phase ^= 1u;
        }
      }
      if (!ok) {
        abort_s = 1;
        atomicExch(&g_error, 1);
        // copies in flight land before the pair leaves: the leader's barriers count both CTAs'
        if (crank == 0)
          for (int j = 0; j < STAGES; ++j) mbar_wait(&full_bar[j], j < next ? pass ^ 1u : pass);
      }
    }
  } else if (warp == 1) {
    // ---- MMA issuer ----
    const uint32_t ring = smem_u32(smem);
    const uint64_t da0 = A_MN ? desc_mn(ring) : umma_desc(ring);
    const uint64_t db0 = B_MN ? desc_mn(ring + kOperandBytes) : umma_desc(ring + kOperandBytes);
    if (crank == 0 && elect_one()) {
      int s = 0, i = 0;
      uint32_t phase = 0;
      int failed = 0;
#pragma unroll 1
      for (int t = pair; t < total && !failed; t += pairs) {
        const Item im = item_of(t, a);
#pragma unroll 1
        for (int ph = 0; ph < phases && !failed; ++ph) {
          // the up product of the high-precision form comes in ranges of kDrain k-steps
          const int range = EPI == kGateUpHp && ph == 1 ? kDrain : im.k1 - im.k0;
#pragma unroll 1
          for (int k0 = im.k0; k0 < im.k1; k0 += range, ++i) {
            const int b = i & 1, k1 = min(k0 + range, im.k1);
            if (!mbar_wait(&tempty_bar[b], ((uint32_t)(i >> 1) & 1u) ^ 1u)) {
              failed = 4;
              break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t acc = tmem_base + (uint32_t)(b * 256);
            uint32_t add = 0;
#pragma unroll 1
            for (int k = k0; k < k1; ++k) {
              if (!mbar_wait(&full_bar[s], phase)) {
                failed = 2;
                break;
              }
              asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
              const uint64_t da = da0 + (uint32_t)s * (kStageBytes >> 4);
              const uint64_t db = db0 + (uint32_t)s * (kStageBytes >> 4);
#pragma unroll
              for (int kk = 0; kk < kStageK / 16; ++kk) {
                mma(acc, da + (A_MN ? 128 : 2) * kk, db + (B_MN ? 128 : 2) * kk, kIdesc, add);
                add = 1;
              }
              commit(&empty_bar[s]);
              if (++s == STAGES) {
                s = 0;
                phase ^= 1u;
              }
            }
            if (failed) break;
            commit(&tfull_bar[b]);
          }
        }
      }
      if (failed) {
        abort_s = 1;
        atomicExch(&g_error, failed);
      }
    }
  } else {
    // ---- epilogue: warp = (lane quarter, column half) ----
    const int q = warp & 3, half = (warp - 2) >> 2;
    unsigned char* buf =
        smem + (size_t)STAGES * kStageBytes + (size_t)(warp - 2) * kBufBytes;
    const uint32_t lane_addr = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(half * 128);
    float shift = 0.f;
    if (EPI == kBwd && a.l1_grad != nullptr) shift = __ldg(a.l1_grad) * a.inv_m;
    int i = 0;  // accumulators taken so far
    auto take = [&]() -> bool {  // waits for accumulator i
      bool ok = mbar_wait(&tfull_bar[i & 1], (uint32_t)(i >> 1) & 1u);
      ok = __all_sync(0xffffffffu, ok);
      // the two warps of a pack's rows meet at barriers: they go on or give up together
      if (kIsPack) ok = named_barrier_and(1 + q, 64, ok);
      if (!ok) {
        abort_s = 1;
        atomicExch(&g_error, 3);
        return false;
      }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      return true;
    };
    auto release = [&]() {  // this warp has read accumulator i
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) arrive_leader(&tempty_bar[i & 1]);
      ++i;
    };
    int parity = 0;
    for (int t = pair; t < total; t += pairs) {
      const Item im = item_of(t, a);
      int mt, nt;
      tile_of(im.tile, m_tiles, a, mt, nt);
      const int row0 = mt * kTile + crank * 128 + q * 32;
      const int row = row0 + lane;
      const bool live = row < rows;
      __nv_bfloat16* out = a.out + (size_t)row * a.ld + nt * kTile + half * 128;
      if (kPlain && a.out_mt > 0 && mt >= a.out_mt) {
        const int o = mt / a.out_mt;
        out = a.out_more[o - 1] + (size_t)(row - o * a.out_mt * kTile) * a.ld + nt * kTile + half * 128;
      }
      uint2 pw[kTrain ? 8 : 1], rw[EPI == kBwd ? 8 : 1];  // the rows' first slab words
      int tail_slot = -1;
      auto load_pattern = [&]() {
        if constexpr (EPI == kMulHp) load_values(a, buf, row0, rows, nt, half, lane);
        if constexpr (kTrain) {
          load_words(a.slab_p, a, row0, rows, nt, 0, lane, pw);
          if (a.row_slot != nullptr && live) tail_slot = a.row_slot[row];
        }
        if constexpr (EPI == kBwd) load_words(a.slab_r, a, row0, rows, nt, 0, lane, rw);
      };
      // the pattern is fetched under the MMAs of this tile (a split tile's only by the warp that
      // finishes it)
      if (im.split_tile < 0) load_pattern();
      if (!take()) break;
      Source src = {lane_addr + (uint32_t)((i & 1) * 256), nullptr, a.splits};

      if (EPI == kStore && a.sums != nullptr) {
        float* dst = a.sums + ((size_t)im.split * rows + row) * a.n_tiles * kTile + nt * kTile + half * 128;
#pragma unroll 1
        for (int cb = 0; cb < 4 && row0 < rows; ++cb) {
          float v[32];
          tmem_ld32(src.acc + (uint32_t)(cb * 32), v);
          if (!live) continue;
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            uint32_t w[16];
#pragma unroll
            for (int p = 0; p < 16; ++p) w[p] = __float_as_uint(v[16 * c + p]);
            store64(reinterpret_cast<__nv_bfloat16*>(dst + cb * 32 + c * 16), w, 1);
          }
        }
        release();
        continue;
      }
      if (!kGate2 && im.split_tile >= 0) {
        const size_t blk = ((size_t)crank * 8 + q * 2 + half) * (128 * 32) + lane;
        float* mine = a.part + (size_t)(im.split_tile * a.splits + im.split) * kItemFloats + blk;
#pragma unroll 1
        for (int cb = 0; cb < 4 && row0 < rows; ++cb) {
          float v[32];
          tmem_ld32(src.acc + (uint32_t)(cb * 32), v);
#pragma unroll
          for (int c = 0; c < 32; ++c) __stcg(mine + cb * 1024 + c * 32, v[c]);
        }
        __threadfence();
        release();
        unsigned int* ctr = a.counters + (im.split_tile * 2 + crank) * 8 + q * 2 + half;
        bool last;
        if (kIsPack) {  // both halves of a row decide together: the slots of the second half follow
          named_barrier(1 + q, 64);
          if (half == 0 && lane == 0) {
            const unsigned int old = atomicAdd(ctr, 1u);
            if (old == (unsigned int)a.splits - 1u) *ctr = 0u;
            last_s[q] = old == (unsigned int)a.splits - 1u;
          }
          named_barrier(1 + q, 64);
          last = last_s[q] != 0;
        } else {
          unsigned int old = 0;
          if (lane == 0) {
            old = atomicAdd(ctr, 1u);
            if (old == (unsigned int)a.splits - 1u) *ctr = 0u;
          }
          last = __shfl_sync(0xffffffffu, old, 0) == (unsigned int)a.splits - 1u;
        }
        if (!last) continue;
        __threadfence();
        src.part = a.part + (size_t)im.split_tile * a.splits * kItemFloats + blk;
        load_pattern();
      }

      uint32_t mask[4];
      int slot = 0, first_slot = 0;
      if (kIsPack) {
        // pass 1: positives of each 32-column block as a mask, bf16 values into the buffer
        int cnt = 0;
#pragma unroll
        for (int cb = 0; cb < 4; ++cb) {
          float v[32];
          fetch32(src, cb, v);
          if (a.bias != nullptr) {
            const float* bp = a.bias + nt * kTile + half * 128 + cb * 32;
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
          mask[cb] = live ? m : 0u;
          cnt += __popc(mask[cb]);
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            uint32_t w[4];
#pragma unroll
            for (int p = 0; p < 4; ++p)
              w[p] = pack2(fmaxf(v[8 * j + 2 * p], 0.f), fmaxf(v[8 * j + 2 * p + 1], 0.f));
            *reinterpret_cast<uint4*>(at(buf, lane, cb * 64 + j * 16)) =
                make_uint4(w[0], w[1], w[2], w[3]);
          }
        }
        if (src.part == nullptr) release();
        // the second half's slots follow the first half's
        slot = 0;
        if (half == 0) half_count[parity][q * 32 + lane] = cnt;
        named_barrier(1 + q, 64);
        if (half == 1) slot = half_count[parity][q * 32 + lane];
        parity ^= 1;
        first_slot = slot;
        const int cap = a.slab_w - 1;
        uint32_t* slab = a.slab_p + (size_t)row * a.row_words + (size_t)nt * a.slab_w;
        if (half == 1 && live) slab[0] = (uint32_t)(slot + cnt);
        if (a.entries != nullptr) {
          const int kept = max(min(slot + cnt, cap) - slot, 0);
          const int sum = __reduce_add_sync(0xffffffffu, kept);
          if (lane == 0 && sum > 0) atomicAdd(a.entries, (unsigned int)sum);
        }
        // pass 2: entries; a value past the slab's capacity leaves the buffer too (unless keep_all)
#pragma unroll
        for (int cb = 0; cb < 4; ++cb) {
          uint32_t m = mask[cb];
          const uint32_t col0 = (uint32_t)(nt * kTile + half * 128 + cb * 32);
          while (m != 0u) {
            const int c = __ffs(m) - 1;
            m &= m - 1;
            uint16_t* p = reinterpret_cast<uint16_t*>(at(buf, lane, cb * 64 + c * 2));
            if (slot < cap) slab[1 + slot] = (col0 + c) | ((uint32_t)*p << 16);
            else if (EPI != kPack && !a.keep_all) *p = 0;
            ++slot;
          }
        }
        __syncwarp();
        if (EPI == kPackDense) {  // what the slab stores, as a dense row
#pragma unroll
          for (int cb = 0; cb < 4; ++cb) {
            uint32_t w[16];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const uint4 g4 = *reinterpret_cast<const uint4*>(at(buf, lane, cb * 64 + j * 16));
              w[4 * j] = g4.x;
              w[4 * j + 1] = g4.y;
              w[4 * j + 2] = g4.z;
              w[4 * j + 3] = g4.w;
            }
            if (live) store64(out + cb * 32, w, a.wide);
          }
        }
        if (!kGate2 || gate_only) continue;
        if constexpr (EPI == kGateUpHp) {  // the up product of the same tile, range by range
          float u[4][32] = {};
          bool ok = true;
#pragma unroll 1
          for (int k = 0; k < a.ksteps; k += kDrain) {
            ok = take();
            if (!ok) break;
            const uint32_t acc = lane_addr + (uint32_t)((i & 1) * 256);
#pragma unroll
            for (int cb = 0; cb < 4; ++cb) {
              float v[32];
              tmem_ld32(acc + (uint32_t)(cb * 32), v);
#pragma unroll
              for (int c = 0; c < 32; ++c) u[cb][c] += v[c];
            }
            release();
          }
          if (!ok) break;
          float* h = a.values + (size_t)row * a.row_words + (size_t)nt * a.slab_w + 1;
#pragma unroll
          for (int cb = 0; cb < 4; ++cb) {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const uint4 g4 = *reinterpret_cast<const uint4*>(at(buf, lane, cb * 64 + j * 16));
              const uint32_t g[4] = {g4.x, g4.y, g4.z, g4.w};
#pragma unroll
              for (int e = 0; e < 8; ++e) {
                const int c = 8 * j + e;
                if ((mask[cb] >> c) & 1u) {
                  if (first_slot < cap) h[first_slot] = (e & 1 ? hi_f(g[e >> 1]) : lo_f(g[e >> 1])) * u[cb][c];
                  ++first_slot;
                }
              }
            }
            __syncwarp();
          }
          continue;
        }
        if (!take()) break;  // the up product of the same tile
        src = Source{lane_addr + (uint32_t)((i & 1) * 256), nullptr, 1};
      }

      if constexpr (kTrain) {
        auto done = [&]() {
          if (src.part == nullptr) release();
        };
        if constexpr (EPI == kFwd) {
          float l1 = forward_tile(a, &map_a1, src, buf, row0, rows, nt, half, lane, pw, tail_slot, done);
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) l1 += __shfl_xor_sync(0xffffffffu, l1, o);
          if (lane == 0)  // one sum of |T| per warp and tile
            a.l1_part[((size_t)im.tile * 2 + crank) * 8 + q * 2 + half] = l1;
        } else {
          backward_tile(a, &map_a1, &map_b1, src, buf, row0, rows, nt, half, lane, pw, rw, tail_slot,
                        shift, done);
        }
      } else if (!kIsPack || EPI == kGateUp) {
#pragma unroll 1
        for (int cb = 0; cb < 4; ++cb) {
          float v[32];
          fetch32(src, cb, v);
          if (EPI == kStoreCarry) {
            float* carry = a.carry + (((size_t)im.tile * 2 + crank) * 8 + q * 2 + half) * (128 * 32) +
                           cb * 1024 + lane;
            if (a.carry_in) {
#pragma unroll
              for (int c = 0; c < 32; ++c) v[c] += __ldcg(carry + c * 32);
            }
            if (a.carry_out) {
#pragma unroll
              for (int c = 0; c < 32; ++c) __stcg(carry + c * 32, v[c]);
              continue;
            }
          }
          if (kPlain) {
            uint32_t w[16];
#pragma unroll
            for (int p = 0; p < 16; ++p)
              w[p] = a.relu ? pack2(fmaxf(v[2 * p], 0.f), fmaxf(v[2 * p + 1], 0.f))
                            : pack2(v[2 * p], v[2 * p + 1]);
            if (live) store64(out + cb * 32, w, a.wide);
          } else if (EPI == kGateUp) {
            uint32_t w[16];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const uint4 g4 = *reinterpret_cast<const uint4*>(at(buf, lane, cb * 64 + j * 16));
              const uint32_t g[4] = {g4.x, g4.y, g4.z, g4.w};
#pragma unroll
              for (int p = 0; p < 4; ++p) {
                const int c = 8 * j + 2 * p;
                const uint32_t m = nonzero2(g[p]);     // never touch u where nothing is stored
                w[4 * j + p] = mul2(g[p], pack2(v[c], v[c + 1]) & m) & m;
              }
            }
            if (live) store64(out + cb * 32, w, a.wide);
          } else if (EPI == kMulHp) {
            uint4 g4[4];
#pragma unroll
            for (int j = 0; j < 4; ++j)
              g4[j] = *reinterpret_cast<const uint4*>(at(buf, lane, cb * 64 + j * 16));
            uint32_t w0[16], w1[16], w2[16];
            mul_hp(g4, v, w0, w1, w2);
            if (live) {
              const size_t h = (size_t)a.n_tiles * kTile;
              store64(out + cb * 32, w0, a.wide);
              store64(out + h + cb * 32, w1, a.wide);
              store64(out + 2 * h + cb * 32, w2, a.wide);
            }
          }
        }
        if (src.part == nullptr) release();
        __syncwarp();
      }
    }
    if (kTrain && lane == 0) tma_store_wait();
  }

  __syncwarp();
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  cluster.sync();
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512)
                 : "memory");
  }
}

// ---- host side -------------------------------------------------------------
struct Operand {
  const void* base;
  int64_t rows, k;   // logical: rows x k; stored [rows][k] (K-major) or [k][rows] (mn)
};

inline int operand_map(CUtensorMap* map, const Operand& o, bool mn) {
  // box of 64 contiguous elements (128 bytes); a pair CTA holds 128 rows: one K-major box of
  // 128 rows, or two MN-major boxes of 64 rows x 64 k
  return mn ? make_map(map, o.base, o.k, o.rows, 64) : make_map(map, o.base, o.rows, o.k, 128);
}

// out = bf16 of the sum over the ranges of k, in their order.
__global__ void __launch_bounds__(256)
sum_ranges_kernel(const float4* __restrict__ sums, uint2* __restrict__ out, int splits, size_t n4,
                  const RunIf run_if) {
  pdl_wait();
  if (run_if.entries != nullptr && !stored_more(run_if)) return;
  const size_t i = (size_t)blockIdx.x * 256 + threadIdx.x;
  if (i >= n4) return;
  float4 v[8];
#pragma unroll
  for (int s = 0; s < 8; ++s)
    if (s < splits) v[s] = __ldcg(sums + (size_t)s * n4 + i);
  float4 t = v[0];
#pragma unroll
  for (int s = 1; s < 8; ++s)
    if (s < splits) {
      t.x += v[s].x;
      t.y += v[s].y;
      t.z += v[s].z;
      t.w += v[s].w;
    }
  out[i] = make_uint2(pack2(t.x, t.y), pack2(t.z, t.w));
}

// How the tiles of the last wave are cut along k: as many equal ranges as still fit the wave, at
// least 4 k-steps each.  A product of less than one wave whose sums go to memory (`all`) takes up
// to 8 ranges, added by a kernel of their own on all SMs; the last wave of another one up to 4,
// added by the warps that arrive last.  Those warps read the sums back in eight dependent rounds, so
// short products are left whole: non-gated MLP, 2 %, us, cut / whole: 16 k-steps (D 1024, H 4096)
// 1200 tokens 59.7 / 51.9; 32 (D 2048, H 8192) 1200 tokens 110 / 106, 3000 tokens 174 / 171;
// 64 (D 4096, H 16384) 640 tokens 181 / 184, 1200 tokens 266 / 270.
constexpr int kCutKsteps = 64;
struct Split {
  int64_t full_tiles;
  int splits;
};
inline Split choose_split(int64_t tiles, int ksteps, int64_t slots, bool all) {
  const int64_t tail = tiles % slots;
  if (tail == 0) return {tiles, 1};
  const bool own_kernel = all && tiles < slots;
  if (!own_kernel && ksteps < kCutKsteps) return {tiles, 1};
  int64_t s = slots / tail;
  if (s > ksteps / 4) s = ksteps / 4;
  if (s > (own_kernel ? 8 : 4)) s = own_kernel ? 8 : 4;
  if (s < 2) return {tiles, 1};
  return {tiles - tail, (int)s};
}
inline size_t split_bytes(const Split& s, int64_t tiles) {
  return s.splits < 2 ? 0 : (size_t)(tiles - s.full_tiles) * s.splits * kTile * kTile * sizeof(float);
}
inline size_t part_bytes(int64_t tiles, int ksteps, int64_t slots, bool all) {
  return split_bytes(choose_split(tiles, ksteps, slots, all), tiles);
}
inline void give_room(Args& a, const SplitRoom& room) {
  a.part = room.part;
  a.part_bytes = room.bytes;
  a.counters = room.counters;
}

template <int EPI, bool A_MN, bool B_MN>
int launch(const char* fn, const Operand& a0, const Operand& a1, const Operand& b0,
           const Operand& b1, Args args, int64_t row_capacity, int sm_count, cudaStream_t stream) {
  constexpr bool kTrain = EPI == kFwd || EPI == kBwd;
  constexpr int STAGES = EPI == kStore || EPI == kStoreCarry ? 6 : EPI == kBwd ? 4 : 5;
  constexpr size_t smem = (size_t)STAGES * kStageBytes + buf_bytes(EPI) + 1024;
  CUtensorMap ma0, ma1, mb0, mb1;
  if (int rc = operand_map(&ma0, a0, A_MN)) return rc;
  if (int rc = operand_map(&mb0, b0, B_MN)) return rc;
  if (kTrain) {  // a1, b1: the dense results, stored in blocks of 32 rows
    if (int rc = make_map(&ma1, a1.base, a1.rows, a1.k, 32)) return rc;
    if (int rc = make_map(&mb1, b1.base, b1.rows, b1.k, 32)) return rc;
  } else {
    if (int rc = operand_map(&ma1, a1, A_MN)) return rc;
    if (int rc = operand_map(&mb1, b1, B_MN)) return rc;
  }
  auto kern = pair_gemm_kernel<EPI, A_MN, B_MN, STAGES>;
  static size_t granted[64] = {0};
  if (int rc = ensure_dynamic_smem(kern, smem, granted, fn)) return rc;
  const int64_t tiles = (row_capacity + kTile - 1) / kTile * args.n_tiles;
  const int64_t slots = sm_count / 2;
  const bool can_sum = EPI == kStore && args.out_mt == 0 && !args.relu &&
                       args.ld == (long long)args.n_tiles * kTile;
  Split sp = EPI != kGateUp && EPI != kGateUpHp && args.part != nullptr && args.counters != nullptr &&
                     args.rows_ptr == nullptr
                 ? choose_split(tiles, args.ksteps, slots, can_sum)
                 : Split{tiles, 1};
  if (split_bytes(sp, tiles) > args.part_bytes) sp = {tiles, 1};
  args.full_tiles = (int)sp.full_tiles;
  args.splits = sp.splits;
  const bool sum_after = can_sum && sp.splits > 1 && sp.full_tiles == 0;
  args.sums = sum_after ? args.part : nullptr;
  const int64_t items = sp.full_tiles + (tiles - sp.full_tiles) * sp.splits;
  const int64_t pairs = items < slots ? items : slots;
  args.group = args.n_tiles >= 10 ? 8 : (int)((slots + args.n_tiles - 1) / args.n_tiles);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(2 * pairs), 1, 1);
  cfg.blockDim = dim3(kThreads, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = add_pdl_attribute(attr, 1);
  cudaError_t e = cudaLaunchKernelEx(&cfg, kern, ma0, ma1, mb0, mb1, args);
  if (e != cudaSuccess) return fail(B200_ECUDA, "%s: launch: %s", fn, cudaGetErrorString(e));
  if (sum_after) {
    const size_t n4 = (size_t)args.rows * args.n_tiles * kTile / 4;
    cudaLaunchConfig_t sum = {};
    sum.gridDim = dim3((unsigned)((n4 + 255) / 256), 1, 1);
    sum.blockDim = dim3(256, 1, 1);
    sum.stream = stream;
    cudaLaunchAttribute sattr[1];
    sum.attrs = sattr;
    sum.numAttrs = add_pdl_attribute(sattr, 0);
    e = cudaLaunchKernelEx(&sum, sum_ranges_kernel, reinterpret_cast<const float4*>(args.sums),
                           reinterpret_cast<uint2*>(args.out), args.splits, n4, args.run_if);
    if (e != cudaSuccess) return fail(B200_ECUDA, "%s: launch: %s", fn, cudaGetErrorString(e));
  }
  return B200_OK;
}

}  // namespace pg
}  // namespace
}  // namespace b200
