// Device kernel launchers for the block-sparse contraction engine (sm_100a).
//
// Every launcher enqueues work on the given stream and returns immediately.
// Offsets are in elements (doubles) relative to the base pointers passed.
#pragma once
#include <algorithm>
#include <cstdint>
#include <cuda_runtime.h>

namespace sb {

// ── grouped FP64 GEMM with segmented accumulation ──────────────────────────
//
// For every C block c:  C_c = sum_{p in [pair_begin_c, pair_end_c)} X_p * Y_p
// where X_p is M_c x K_p and Y_p is K_p x N_c, C_c is column-major M_c x N_c
// (leading dimension M_c).  X is read "N" (element (i,k) at x + i + k*ldx) or
// "T" (element (i,k) at x + k + i*ldx); Y likewise ((k,j) at y + k + j*ldy or
// y + j + k*ldy).  Each C tile is produced by exactly one CTA: no atomics, C
// is written once (no zero-init needed), accumulation order over pairs is the
// pair order.
// Tiles of C block c are CTAs [tile_begin, tile_begin + mtiles*ntiles); the
// kernel finds its C block by binary search over tile_begin, so no per-tile
// descriptor list is built or uploaded.
// ldc: column stride of the C block in C.  It equals M except for the edge
// sub-blocks of launch_gemm_f64_edges (a row range of a larger block); the
// thin kernels with small rows (small_rows) require ldc == M.  tshape: tile shape of the block in
// launch_gemm_f64_edges (0 = 64x64, 1 = 64x32, 2 = 32x64, 3 = 64x48,
// 4 = 48x64), else 0.
struct GemmCBlock {
  int64_t c_off;
  int32_t M, N;
  int32_t pair_begin, pair_end;
  int32_t tile_begin, mtiles;
  int32_t ldc, tshape;
};
struct GemmPair {
  int64_t x_off, y_off;
  int32_t K, ldx, ldy, pad;
};

// CTA tile shapes with 32x32 warp tiles, k-tile 16, 3 stages, plus T64x32.
// Measured on the H_eff steps (chi = 2048): 32x64 / 64x32 warp tiles need
// 190-250 registers, halve the resident CTAs and run 4-16% slower; 4 stages,
// k-tile 32 and eight 32x16 warps run 0-18% slower on the psi*L step.
// T64x32: four 32x16 warps, 4 stages, used for the few-tile, long-K launches
// that otherwise go to split-K (H_eff R*T3: 2.17 against 2.26 ms).
enum class GemmShape : int { T64x64 = 0, T128x32 = 1, T32x128 = 2, T128x64 = 3, T64x128 = 4, T64x32 = 5 };

// splitk > 1 (at most kMaxSplitK): the concatenated K range of every C tile is
// cut into splitk segments, each computed by a CTA of its own, and summed in
// segment order (deterministic): through the shared memory of a cluster, or,
// with partial (splitk * ntiles * BM*BN doubles), by a second kernel.
constexpr int kMaxSplitK = 16, kPortableCluster = 8;
cudaError_t launch_gemm_f64(const double* X, const double* Y, double* C,
                            const GemmCBlock* d_cblocks, int32_t ncblocks, const GemmPair* d_pairs,
                            int64_t ntiles, bool xT, bool yT, GemmShape shape, cudaStream_t s,
                            int splitk = 1, double* partial = nullptr);

// Tiled GEMM over C sub-blocks of five tile shapes in one launch: each
// GemmCBlock's tshape gives its tile (0 = 64x64; 1 = 64x32 and 3 = 64x48 for
// column edges of width <= 32 and <= 48; 2 = 32x64 and 4 = 48x64 for row
// edges of height <= 32 and <= 48); tiles are
// numbered through tile_begin / mtiles of that shape.  Sub-blocks carry their
// own ldc and pairs whose offsets start at the sub-block's first row and
// column.  partial, if any: splitk * ntiles * 4096 doubles.
cudaError_t launch_gemm_f64_edges(const double* X, const double* Y, double* C, const GemmCBlock* d_cblocks,
                                  int32_t ncblocks, const GemmPair* d_pairs, int64_t ntiles, bool xT, bool yT,
                                  cudaStream_t s, int splitk = 1, double* partial = nullptr);

// Thin variant for launches whose every pair has K <= 16 and whose C blocks
// have min(M, N) <= 16 (HBM-bound): DMMA on 128 x 16 strips of the long side,
// cp.async double buffering across pairs.  Strips of C block c:
// [tile_begin, tile_begin + ceil(long/128)) when mtiles == 1; a group of S
// consecutive blocks with equal long extent, each carrying the group's
// tile_begin and mtiles = S, takes strips in turn (strip s of member j is
// tile_begin + s*S + j).  persistent: a
// grid of 5 CTAs per SM walks the strips with the copy pipeline running
// across strip boundaries and stores C from the fragments (needs >= 1 pair
// per C block); otherwise one CTA per strip with shared-memory staged stores.
// long_f32: the long operand (Y when small_rows, else X) and C hold FP32
// values (the intermediates of the tensor-core H_eff chain); the small
// operand stays FP64 and the arithmetic FP64.  Persistent kernel only.
cudaError_t launch_gemm_f64_skinny(const double* X, const double* Y, double* C,
                                   const GemmCBlock* d_cblocks, int32_t ncblocks, const GemmPair* d_pairs,
                                   int64_t nctas, bool xT, bool yT, bool small_rows, int small_max,
                                   int k_max, cudaStream_t s, bool persistent = false, bool long_f32 = false);

// Number of tiles of a (M, N) C block for the given tile shape.
void gemm_tile_dims(GemmShape shape, int* bm, int* bn);

// ── the same grouped GEMM on the tcgen05 tensor cores (sb_gemm_tc.cu) ─────
//
// FP32 operands (X, Y: element offsets as in GemmPair), arithmetic in TF32
// with FP32 accumulation, result FP64 (c_f64) or FP32.  passes = 3 splits
// every operand into TF32 hi + lo parts and sums a_hi*b_lo + a_lo*b_hi +
// a_hi*b_hi (about 22 significant bits per operand), passes = 1 multiplies
// the TF32-rounded operands once.
// Work items are listed explicitly: item i covers rows [a0, a0 + 128) of the
// A side and [b0, b0 + nb) of the B side of C block cb (nb a multiple of 16
// in 16..256), and nkt k-tiles (32 deep) of its C block's concatenated pair
// K ranges starting at pair p0, offset k0 (a multiple of 32).  Without swap
// the A side is X (rows of C) and the B side Y (columns of C); with swap the
// other way round.  An item with part < 0 covers the whole K range and
// writes C; part >= 0 marks a k-segment of a split tile, written in FP64 to
// partial tile `part` (column-major 128 x 256 doubles) and summed in segment
// order into C by the reduction that follows (one TcSplit per split tile:
// its geometry and its parts [part0, part0 + nparts)).  Items [nz_begin,
// ntiles) belong to C blocks without pairs and are written as zeros.  Within
// an item the k-tiles accumulate in FP32 chunks of kc k-tiles (the tensor
// core's accumulation error grows with the chunk length) whose sum is formed
// in FP32 with round-to-nearest adds.  fold must be set when an item has
// more than kc k-tiles (one accumulator and the running sum in TMEM; without
// it two accumulators alternate and every item is one chunk).  A persistent grid of one CTA per SM walks the list
// with stride gridDim.x, so the list order (the host sorts by work) balances
// the load.  *d_status is set to 1 if a bounded wait on the tensor core ran
// out (the results are then invalid).
struct TcTile {
  int32_t cb, a0, b0, nb;
  int32_t p0, k0, nkt, part;
};
struct TcSplit {
  int32_t cb, a0, b0, nb;
  int32_t part0, nparts, pad0, pad1;
};
constexpr int kTcMaxN = 256;
constexpr int64_t kTcPartElems = 128 * kTcMaxN;  // doubles of one partial tile
// Operands arrive packed (launch_tc_pack): per pair p, packs[p] locates the
// images of its A-side block (a_base: 128-row tiles, nkt k-tiles each, 32 KB
// per k-tile: hi plane then lo plane) and of its B-side block (b_base: tiles
// of nbs rows, 2*nbs*128 bytes per k-tile); item rows a0 and b0 select the
// tile (a0 / 128, b0 / nbs).
struct TcPack {
  int64_t a_base, b_base;
  int32_t nkt, nbs;
};
cudaError_t launch_gemm_tc(const void* pack_a, const void* pack_b, void* C, bool c_f64, const GemmCBlock* d_cblocks,
                           const GemmPair* d_pairs, const TcPack* d_packs, const TcTile* d_tiles, int32_t ntiles,
                           int32_t nz_begin, bool swap, int passes, int kc, bool fold, double* d_partial,
                           const TcSplit* d_splits, int32_t nsplits, int* d_status, cudaStream_t s);
// One packed k-tile image of one operand tile: rows [0, rows) x k [0, kv)
// (element (r, k) at src + r*ld + k when kc, else src + r + k*ld; elements of
// the FP64 or FP32 operand array), zero elsewhere, written at byte dst as the
// hi plane and (passes = 3) the lo plane plane bytes further; plane = image
// rows x 128 bytes in the K-major 128-byte-swizzled layout the tensor core
// reads.
struct TcImage {
  int64_t src, ld, dst;
  int32_t rows, kv, plane, kc;
};
cudaError_t launch_tc_pack(const void* src, bool src_f64, const TcImage* d_imgs, int64_t nimg, void* dst, int passes,
                           cudaStream_t s);

// ── the same grouped GEMM in FP64 through 8-bit integer products ───────────
// (sb_gemm_i8.cu: tcgen05 kind::i8).  X is the 128-row side, Y the other.
// Scratch holds the packed digit planes, one scale word per operand row
// (zeroed before the packs) and a flag (zeroed too): the kernels set it when
// an operand row's magnitude is outside 2^+-400 (or not finite), or when a
// bounded wait ran out; C is then what launch_gemm_f64_fallback, which must
// follow on the stream, computes.
//
// C blocks whose pairs read the same Y blocks (the same offsets, leading
// dimensions and K in the same order) form one group and share row tiles: their
// rows are numbered through, and row_off / row_ld give each row's C offset and
// column stride.
struct I8Group {
  int32_t rows, N, row0, pad;  // row0: the group's first entry in the row tables
};
// A piece of a 128-row (X) or rows_img-row (Y) x 64 k-tile image: image rows
// [row0, row0 + rows) are an operand block's, element (r, k) at src + r*ld + k
// when kc, else src + r + k*ld, kv <= 64 of them along k; rows up to row_end and
// the rest of k are zeros.  Seven planes of rows_img * 64 bytes at byte dst; the
// scale of row row0 at index scale.  With strip_k > 0 an entry is a strip: rows
// of an aligned range of 16 image rows and all of K (kv <= strip_k <=
// kI8StripK), its k-tiles' images one after the other.
struct I8Image {
  int64_t src, ld, dst;
  int32_t scale, row0, rows, row_end, rows_img, kv, kc, pad;
};
constexpr int32_t kI8StripK = 768;  // 16 rows of 768: two CTAs per SM
// An operand block in its stack of rows: element (r, k) at src + r*ld + k when
// kc, else src + r + k*ld; stack rows [at, at + rows) of total; the stack's
// images from byte dst, its scales from index scale; the block's entries of the
// image list begin at first.
struct I8Block {
  int64_t src, ld, dst;
  int32_t scale, at, rows, total, tile, K, kc, strip, first, pad;
};
// Entries of a block, and its p-th: strips in row order, k-tiles row tile by row
// tile.  Lists are written on the device, 56 bytes an entry from one block
// descriptor: at chi = 2048 R*T3 has 14000 and their upload cost milliseconds.
__host__ __device__ inline int32_t i8_entries(const I8Block& b) {
  if (b.rows <= 0) return 0;
  const int32_t unit = b.strip ? 16 : b.tile;
  return ((b.at + b.rows - 1) / unit - b.at / unit + 1) * (b.strip ? 1 : (b.K + 63) / 64);
}
__host__ __device__ inline I8Image i8_entry(const I8Block& b, int32_t p) {
  const int32_t nkt = (b.K + 63) / 64, unit = b.strip ? 16 : b.tile, per = b.strip ? 1 : nkt;
  const int32_t u0 = (b.at / unit + p / per) * unit, kt = p % per;
  const int32_t lo = b.at > u0 ? b.at : u0, hi = b.at + b.rows < u0 + unit ? b.at + b.rows : u0 + unit;
  const int32_t t = lo / b.tile, r = lo - t * b.tile, left = b.K - 64 * kt;
  const int64_t dr = lo - b.at, dk = 64 * kt;
  return I8Image{b.src + (b.kc ? dr * b.ld + dk : dr + dk * b.ld),
                 b.ld,
                 b.dst + (static_cast<int64_t>(t) * nkt + kt) * 7 * 64 * b.tile,
                 b.scale + lo,
                 r,
                 hi - lo,
                 hi == b.total ? b.tile : r + hi - lo,
                 b.tile,
                 b.strip ? b.K : left < 64 ? left : 64,
                 b.kc,
                 0};
}
cudaError_t launch_i8_entries(const I8Block* d_blocks, int64_t nblocks, I8Image* d_imgs, cudaStream_t s);
// Row tables of launch_gemm_i8 from the C blocks: rows [row0, row0 + M) are
// C's at c_off, column stride ldc.
struct I8RowRun {
  int64_t c_off;
  int32_t ldc, M, row0, pad;
};
cudaError_t launch_i8_rows(const I8RowRun* d_runs, int64_t nruns, int64_t* d_row_off, int32_t* d_row_ld,
                           cudaStream_t s);
cudaError_t launch_i8_pack(const double* src, const I8Image* d_imgs, int64_t nimg, int32_t strip_k, uint32_t* d_rowhi,
                           void* dst, int* d_flag, cudaStream_t s);
// Per pair: byte offsets of the images of its X block (row tiles of 128, nkt
// k-tiles each) and Y block (column tiles of nbs), and the scale indices of
// their first row and column.
struct I8Pack {
  int64_t a_base, b_base;
  int32_t a_sc, b_sc, nkt, nbs;
};
constexpr int kI8MaxN = 128;
constexpr int64_t kI8PartElems = 128 * kI8MaxN;  // doubles of one partial tile
// k-tiles per INT32 accumulation chunk: 24 * 64 = 1536 terms keep the four
// diagonals that are combined (5 * 1536 * 2^14 * 2^24 + ...) below 2^51.
constexpr int kI8Chunk = 24;
// Items, splits and pair-less items as for launch_gemm_tc, with 64-deep
// k-tiles, tiles of 128 x nb (nb <= 128) and column-major 128 x 128 partials.
// A tile's cb is its group's index.  CTA i of the nctas (one per SM at most)
// runs items [first[i], first[i + 1]).
cudaError_t launch_gemm_i8(const void* pack, double* C, const I8Group* d_groups, const int64_t* d_row_off,
                           const int32_t* d_row_ld, const I8Pack* d_packs, const uint32_t* d_rowhi,
                           const TcTile* d_tiles, const int32_t* d_first, int32_t nctas, int32_t ntiles,
                           int32_t nz_begin, double* d_partial, const TcSplit* d_splits, int32_t nsplits, int* d_flag,
                           cudaStream_t s);
// The DMMA kernel over the same C blocks (64x64 tiles numbered by tile_begin),
// on a grid that returns at once unless *d_flag is set (NULL: it always runs).
cudaError_t launch_gemm_f64_fallback(const double* X, const double* Y, double* C, const GemmCBlock* d_cblocks,
                                     int32_t ncblocks, const GemmPair* d_pairs, int64_t ntiles, bool xT, bool yT,
                                     const int* d_flag, cudaStream_t s);

// ── outer-product accumulation (K = 1 pairs) on CUDA cores ─────────────────
//
// For every C block c: C_c[i + j*M] = sum_p a_p[i] * b_p[j] in pair order, with
// the reference's rounding (c = c + a*b, no fusion) or Kahan compensation.
struct OuterCBlock {
  int64_t c_off;
  int32_t M, N;
  int32_t pair_begin, pair_end;
};
struct OuterPair {
  int64_t a_off, b_off;
};
cudaError_t launch_outer_acc(const double* Abase, const double* Bbase, double* C,
                             const OuterCBlock* d_cblocks, int64_t ncblocks,
                             const OuterPair* d_pairs, int64_t max_elems, bool kahan,
                             cudaStream_t s);

// ── segmented scaled accumulation (axpy) ───────────────────────────────────
//
// For every segment g: C[c_off_g + t] = sum_{e in seg g} alpha_e * src[src_off_e + t]
// for t < len_g, rounding as c = c + alpha*src (alpha from d_alpha[alpha_idx_e],
// or 1.0 when alpha_idx_e < 0).
struct AxpySeg {
  int64_t c_off;
  int64_t len;
  int32_t e_begin, e_end;
};
struct AxpyEntry {
  int64_t src_off;
  int64_t alpha_idx;
};
cudaError_t launch_axpy_seg(const double* src, const double* d_alpha, double* C,
                            const AxpySeg* d_segs, int64_t nsegs, const AxpyEntry* d_entries,
                            int64_t max_len, cudaStream_t s);

// ── permutes ───────────────────────────────────────────────────────────────
//
// dst block b (packed at b*blk) = tail-permute of src block at src_off[b].
// out_dims[r]: output tail dims (fastest first); in_strides[r]: stride in the
// source block of output axis r.
constexpr int kMaxRank = 12;
struct PermDesc {
  int rank;
  int64_t out_dims[kMaxRank];
  int64_t in_strides[kMaxRank];
};
cudaError_t launch_permute_blocks(const double* src, double* dst, const int64_t* d_src_off,
                                  int64_t nblocks, int64_t blk, const PermDesc& desc,
                                  cudaStream_t s);

// Variable-size block copy: dst[dst_off[i] + e] = src[src_off[i] + e] for e < len[i].
struct BlockCopy {
  int64_t src_off, dst_off, len;
};
cudaError_t launch_copy_blocks(const double* src, double* dst, const BlockCopy* d_items, int64_t n,
                               int64_t max_len, cudaStream_t s);
// Per-block tail permute / pad / crop: output block i (dst_off, out_dims) element
// e reads src[src_off + sum_r c_r * in_strides[r]] when every coordinate c_r is
// below in_lim[r], and writes 0 otherwise (zero padding).
struct BlockPerm {
  int64_t src_off, dst_off, len;
  int rank;
  int64_t out_dims[kMaxRank];
  int64_t in_strides[kMaxRank];
  int64_t in_lim[kMaxRank];
  // division by out_dims[r] (blocks below 2^31 elements) as a multiply and a
  // shift: q = (mulhi(n, div_mul) + n) >> div_shift, exact for n < 2^31
  // (Granlund and Montgomery 1994); set by Divisors
  uint32_t div_mul[kMaxRank], div_shift[kMaxRank];
};
// The divisors of a list of items; short extents, which repeat from block to
// block, are divided out once (400 blocks of three axes: 10 us of host time less).
struct Divisors {
  uint32_t memo[1024] = {};  // div_mul by extent, 0 = not known yet (it is at least 1)
  void set(BlockPerm& b) {
    for (int r = 0; r < b.rank; ++r) {
      const uint64_t d = static_cast<uint64_t>(b.out_dims[r]);
      const uint32_t s = d <= 1 ? 0 : std::min(32u, 64u - static_cast<uint32_t>(__builtin_clzll(d - 1)));
      uint32_t* const m = d < 1024 ? &memo[d] : nullptr;
      b.div_shift[r] = s;
      b.div_mul[r] = m && *m ? *m
                     : d < 1 || d >= (uint64_t{1} << 31)
                         ? 0
                         : static_cast<uint32_t>((uint64_t{1} << 32) * ((uint64_t{1} << s) - d) / d + 1);
      if (m) *m = b.div_mul[r];
    }
  }
};
cudaError_t launch_perm_blocks(const double* src, double* dst, const BlockPerm* d_items, int64_t n,
                               int64_t max_len, cudaStream_t s);
// The same through shared-memory tiles, for items that neither pad nor crop.
// perm_tile_item makes an item's geometry and its number of tiles, or returns
// false when it does not qualify (limits below the output extents, 2^31
// elements or more, no axis to read contiguously); cap = elements of shared memory per tile (perm_tile_cap:
// 1056 to 4160 by the elements moved, so that small operands make enough tiles
// for the chip).  The caller sets tile_begin = tiles before the item; total =
// all tiles.
struct PermTileItem {
  int64_t src_off, dst_off, tile_begin;
  int32_t rank, q;  // q: the output axis that is contiguous in the source
  uint32_t dv, du, tv, tu, tiles_u, tiles_v;
  uint32_t dims[kMaxRank], strides[kMaxRank];
};
constexpr int kPermTileElems = 64 * 65;  // largest cap
constexpr int kPermTileRows = 1024;      // largest tv
inline uint32_t perm_tile_cap(int64_t elems) {
  const int64_t c = elems / (148LL * 12);
  return static_cast<uint32_t>(c < 1056 ? 1056 : c > kPermTileElems ? kPermTileElems : c);
}

inline bool perm_tile_item(const BlockPerm& b, uint32_t cap, PermTileItem* out, int64_t* tiles) {
  if (b.len <= 0 || b.len >= (int64_t{1} << 31) || b.rank < 1) return false;
  PermTileItem p{};
  p.src_off = b.src_off;
  p.dst_off = b.dst_off;
  p.rank = b.rank;
  p.q = b.rank - 1;
  for (int r = b.rank - 1; r >= 0; --r) {
    if (b.in_lim[r] < b.out_dims[r] || (b.out_dims[r] > 1 && b.in_strides[r] >= (int64_t{1} << 31))) return false;
    p.dims[r] = static_cast<uint32_t>(b.out_dims[r]);
    p.strides[r] = b.out_dims[r] > 1 ? static_cast<uint32_t>(b.in_strides[r]) : 0;
    if (b.in_strides[r] == 1 && b.out_dims[r] > 1) p.q = r;
  }
  if (b.len > 1 && (b.out_dims[p.q] == 1 || b.in_strides[p.q] != 1)) return false;
  // output axis 0 contiguous in the source too (crops, outer-axis reorders):
  // a tile would hold one row of axis 0, so only long rows qualify
  if (p.q == 0 && p.dims[0] < 256 && b.len > p.dims[0]) return false;
  // a tile row's source offset is a 32-bit sum; the strides may be those of a
  // longer block, of which these are a part
  int64_t reach = 0;
  for (int r = 0; r < p.q; ++r) reach += (b.out_dims[r] - 1) * static_cast<int64_t>(p.strides[r]);
  if (reach >= (int64_t{1} << 31)) return false;
  int64_t nbatch = 1;
  p.dv = 1;
  for (int r = 0; r < p.q; ++r) p.dv *= p.dims[r];
  p.du = p.dims[p.q];
  for (int r = p.q + 1; r < b.rank; ++r) nbatch *= p.dims[r];
  // about square; a short side is covered whole and the other takes what is
  // left of cap; equal parts, so that no tile is a sliver
  uint32_t side = 24;
  while ((side + 8) * (side + 9) <= cap && side < 64) side += 8;
  uint32_t tv = std::min(p.dv, side), tu = cap / (tv | 1);
  if (p.du < tu) {
    tu = p.du;
    tv = std::min<uint32_t>((cap / tu - 1) | 1, kPermTileRows);
  } else if (tv == side) {
    tu = side;
  }
  tv = std::min(tv, p.dv);
  p.tiles_u = (p.du + tu - 1) / tu;
  p.tiles_v = (p.dv + tv - 1) / tv;
  p.tu = (p.du + p.tiles_u - 1) / p.tiles_u;
  p.tv = (p.dv + p.tiles_v - 1) / p.tiles_v;
  *out = p;
  *tiles = static_cast<int64_t>(p.tiles_u) * p.tiles_v * nbatch;
  return true;
}
cudaError_t launch_perm_block_tiles(const double* src, double* dst, const PermTileItem* d_items, int64_t n,
                                    int64_t total, uint32_t cap, cudaStream_t s);
// The same for items whose out_dims[0] has in_strides[0] == 1 (one warp per
// row of out_dims[0]); max_rows = the largest len / out_dims[0].
cudaError_t launch_perm_block_rows(const double* src, double* dst, const BlockPerm* d_items, int64_t n,
                                   int64_t max_rows, cudaStream_t s);
// ext[b*n2 + r] = smallest axis-r extent of block b (payload at d_off[b],
// extents d_dims[b*n2 ..]) that keeps all its nonzero entries, 0 for a block of
// zeros (d_ext holds 0s on entry).  The scan runs in warp tasks: block b has
// block_extent_tasks(d0, cols, ...) of them (d0 = its first extent, cols =
// the product of the others), starting at d_task_begin[b]; d_task_begin has
// nblocks + 1 entries, the last = ntasks.  budget: elements per task, 512 to
// 8192 by the number of elements scanned (block_extent_budget), the same
// value for every call of one launch.
int64_t block_extent_budget(int64_t elems);
int64_t block_extent_tasks(int64_t d0, int64_t cols, int64_t budget);
cudaError_t launch_block_extents(const double* src, const int64_t* d_off, const int64_t* d_dims,
                                 const int64_t* d_task_begin, int64_t nblocks, int64_t ntasks, int n2,
                                 int64_t budget, int* d_ext, cudaStream_t s);
// The same for blocks below 2^31 elements with tails of at most four axes
// (n2 = the most any block has; dims beyond a block's own n2 are 1), of any
// number of tensors in one launch: tasks are runs of `budget` elements, block
// b's starting at task_begin, its results at ext[ext0 ..] (0 = all zero).
struct ExtBlock {
  const double* p;
  int64_t task_begin;
  uint32_t dims[4];
  int32_t ext0, n2;
};
cudaError_t launch_block_extents_linear(const ExtBlock* d_blocks, int64_t nblocks, int64_t ntasks, int n2,
                                        int64_t budget, int* d_ext, cudaStream_t s);
// flags[i] = 1 if block i of src holds a nonzero outside its box in_lim
// (used to check that cropping a padded block loses nothing).
cudaError_t launch_outside_nonzero(const double* src, const BlockPerm* d_items, int64_t n, int64_t max_len,
                                   uint8_t* flags, cudaStream_t s);

// ── value-dependent structure helpers ──────────────────────────────────────
// flags[b*nslices + s] = any(src[off_b + s*chunk + t] != 0, t < chunk)
cudaError_t launch_slice_nonzero(const double* src, const int64_t* d_off, int64_t nblocks,
                                 int64_t nslices, int64_t chunk, uint8_t* flags, cudaStream_t s);
// flags[q] = any(alpha[ai_q] * src[off_q + t] != 0, t < chunk)
cudaError_t launch_scaled_slice_nonzero(const double* src, const double* alpha,
                                        const int64_t* d_off, const int64_t* d_ai, int64_t n,
                                        int64_t chunk, uint8_t* flags, cudaStream_t s);
// flags[b] = max_t |src[b*blk + t]| > tol
cudaError_t launch_block_max_gt(const double* src, int64_t nblocks, int64_t blk, double tol,
                                uint8_t* flags, cudaStream_t s);
// flags[i] = |src[i]| > atol + rtol*|src[i]|
cudaError_t launch_elem_keep(const double* src, int64_t n, double atol, double rtol,
                             uint8_t* flags, cudaStream_t s);
// max |src[i]| into *d_out (single value)
cudaError_t launch_maxabs(const double* src, int64_t n, double* d_out, cudaStream_t s);

// ── gathers / scatters ─────────────────────────────────────────────────────
cudaError_t launch_gather(const double* src, const int64_t* d_idx, int64_t n, double* dst,
                          cudaStream_t s);
cudaError_t launch_scatter(const double* src, const int64_t* d_idx, int64_t n, double* dst,
                           cudaStream_t s);
// dst[b*blk + t] = scal[b] * src[tmpl_off[b] + t]
cudaError_t launch_scale_blocks(const double* src, const int64_t* d_tmpl_off,
                                const double* d_scal, int64_t nblocks, int64_t blk,
                                double* dst, cudaStream_t s);
// dense[lin_b + stride*t] = data[b*blk + t]
cudaError_t launch_blocks_to_strided(const double* data, const int64_t* d_lin, int64_t nblocks,
                                     int64_t blk, int64_t stride, double* dense, cudaStream_t s);

// ── vector-space operations (Krylov solvers) ───────────────────────────────
// Dot product over chunks of at most kDotChunk elements: *out = sum over
// chunks of sum_t (s*X[x_off+t]) * (s*Y[y_off+t]) with s = S[s_idx] (s = 1
// when s_idx < 0).  d_chunks NULL: the chunks of one contiguous segment of n
// elements.  d_partial holds nchunks doubles; *d_counter is zero before the
// launch and after it; out is device or mapped host memory.  Fixed reduction
// order: identical bits on every call.
constexpr int kDotChunk = 1024;  // 4 elements per thread of a 256-thread CTA
struct DotChunk {
  int64_t x_off, y_off;
  int64_t s_idx;
  int32_t len, pad;
};
cudaError_t launch_dot(const double* X, const double* Y, const double* S, const DotChunk* d_chunks, int64_t nchunks,
                       int64_t n, double* d_partial, unsigned* d_counter, double* out, cudaStream_t s);
// Elementwise R[i] = f(R[i], A[i]) for i < n.
enum MapOp : int { kMapAxpy = 0, kMapAxpby = 1, kMapCopy = 2, kMapMul = 3, kMapScale = 4, kMapFill = 5 };
cudaError_t launch_map(double* R, const double* A, int64_t n, int op, double alpha, double beta, cudaStream_t s);
// Key-union add: C[c_off + e] = A-block, 0 + B-block, or A-block + B-block
// (a_off / b_off < 0 marks a missing operand block).
struct AddBlock {
  int64_t a_off, b_off, c_off, len;
};
cudaError_t launch_add_blocks(const double* A, const double* B, double* C, const AddBlock* d_items, int64_t n,
                              int64_t max_len, cudaStream_t s);

// ── block factorisations (QR, SVD truncation) ──────────────────────────────
// In-place Householder QR of the column-major m x n matrix M (LAPACK dlarfg
// convention): R in the upper triangle, reflector j below the diagonal of
// column j; tau (householder_scalars(m, n) doubles) receives the reflectors'
// scales: the panels' T matrices up to 1024 rows, else one per reflector;
// *launches counts the kernels issued.
int64_t householder_scalars(int64_t m, int64_t n);
cudaError_t launch_householder_qr(double* M, int64_t m, int64_t n, double* tau, cudaStream_t s, int64_t* launches);
// Thin Q (m x k, column-major) from the reflectors in M.
cudaError_t launch_householder_form_q(const double* M, int64_t m, int64_t k, const double* tau, double* Q,
                                      cudaStream_t s, int64_t* launches);
// R (k x n, column-major) = upper triangle of the first k rows of M.
cudaError_t launch_upper(const double* M, int64_t m, int64_t k, int64_t n, double* R, cudaStream_t s);
// Strided 2-D copies: dst[dst_off + r*dst_rs + c*dst_cs] = src[src_off + r*src_rs + c*src_cs]
// (times scale[s_idx + c] when s_idx >= 0) for r < rows, c < cols.
struct Gather2D {
  int64_t src_off, dst_off, rows, cols, src_rs, src_cs, dst_rs, dst_cs, s_idx;
};
cudaError_t launch_gather_2d(const double* src, double* dst, const double* scale, const Gather2D* d_items, int64_t n,
                             int64_t max_elems, cudaStream_t s);
// One-sided Jacobi SVD of row-major m x n matrices (m <= kSvdMaxRows) at
// A + a_off: on return Vt + a_off holds the right singular vectors as rows,
// U + u_off the left ones (column-major m x m) and S + s_off the m singular
// values, all sorted by decreasing singular value.  A is overwritten.
// *d_status is set to 1 when some matrix has not converged in max_sweeps.
constexpr int kSvdMaxRows = 32;
struct SvdGroup {
  int64_t a_off;
  int64_t n;
  int64_t u_off, s_off;
  int32_t m, pad;
};
cudaError_t launch_svd_rows(double* A, double* Vt, double* U, double* S, const SvdGroup* d_groups, int64_t ngroups,
                            int max_sweeps, int* d_status, cudaStream_t s);

// ── scalar programs (aliased bookkeeping) ──────────────────────────────────
// out[g] = sum_{e in seg g} (sa[ia_e] * (ib_e >= 0 ? sb[ib_e] : 1)), left to right.
struct ScalarTerm {
  int64_t ia, ib;
};
cudaError_t launch_scalar_prog(const double* sa, const double* sb, const ScalarTerm* d_terms,
                               const int32_t* d_seg_begin, int64_t nsegs, double* out,
                               cudaStream_t s);

}  // namespace sb
