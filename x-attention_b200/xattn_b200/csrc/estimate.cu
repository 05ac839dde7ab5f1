// Phase 1 of the XAttention prefill path: antidiagonal block-importance estimate.
//
//   S'[i,j] = scale * sum_{t<S} Q[S*i + S-1-t, :] . K[S*j + t, :]        (one row/col = S tokens)
//   P = row softmax of S' over the row's visible columns
//   attn_sums[qb,kb] = sum of P over the (block/S) x (block/S) cell
//
// Reference: xattn/src/Xattention.py:71-136,174-252 (torch branch) and xattn/src/kernels.py:5-156,
// 197-235 (Triton kernels).  Here the S' matrix never exists in memory:
//
//   est_setup_kernel     per 128-row tile, the range of 256-column tiles that hold visible columns
//   est_gemm_kernel      persistent, warp-specialised tcgen05 GEMM.  One thread streams the
//                        stride-reshaped operands with TMA (the reshape is a 5-D tensor map: a row of
//                        the A tile for K-step t is token S*i+S-1-t, of the B tile token S*j+t), one
//                        thread issues 128x256x16 MMAs into a double-buffered TMEM accumulator, four
//                        warps run the epilogue: per row, max over the tile's visible columns, exp2,
//                        sums over groups of block/S columns.  Output per (row, key block): an
//                        un-normalised partial sum, plus the max it was taken against per (row, tile).
//   est_blocksum_kernel  per row tile: the rows' maxima and sums over their column tiles, then per key block: normalise and
//                        add the block/S rows.  (Rows of a single tile need neither, see est_epilogue_row_direct.)
#include <math.h>

#include <type_traits>

#include "select_row.cuh"

namespace xb {

constexpr int kTileM = 128;
constexpr int kTileN = 256;                                  // widest column tile; EstGeom::tile_n is 256 or 128
constexpr int kTileK = 64;                                   // elements per TMA box row = 128 bytes
constexpr int kStages = 4;
constexpr int kMaxStages = 6;                                // stages of the kernels whose stage is 32 KiB
constexpr int kABytes = kTileM * kTileK * 2;                 // 16 KiB
constexpr int kBBytes = kTileN * kTileK * 2;                 // 32 KiB
constexpr int kStageBytes = kABytes + kBBytes;               // 48 KiB
constexpr int kGemmThreads = 192;                            // warp 0 TMA, warp 1 MMA, warps 2-5 epilogue
constexpr int kGemmSmem = kStages * kStageBytes + 1024 /*barriers*/ + 1024 /*alignment slack*/;

// fp32 operands: units of 128 rows x 32 columns go through a ring, four warps split them into three bf16 terms that are kept
// the way a stage of 16-bit operands is, for 64 columns (half of them worked on by the MMAs, half written)
constexpr int kF32Cols = 32;
constexpr int kF32Unit = kTileM * kF32Cols * 4;              // 16 KiB
constexpr int kF32Smem = 224 * 1024;                         // terms and ring: 3 x 32 KiB and 8 units, or 3 x 48 KiB and 5
constexpr int kMaxUnits = 8;
// Warps that split the units, every warp some rows of each: sixteen of up to 88 registers, or, where the epilogue has registers of its own,
// eight of 128, with which the sixteen warps of the CTA make up the register file.
__host__ __device__ constexpr int convert_warps(int direct) { return direct ? 8 : 16; }
// Where the epilogue needs the registers it is a warpgroup of its own (warps 4-7), which takes over what the loading and issuing warps
// (0-3) do not need; the converters follow.  (With 128 registers for all it stored 832 to 2750 bytes per thread to local memory, which is
// L2 here, behind the last product of every tile.  fp32 inputs, 32 heads, estimate and mask, us: 2048 tokens at stride 8 52.2 -> 46.5,
// 3000 at stride 16 in one chunk 80.0 -> 73.1, 4096 81.3 -> 76.0, 1003 30.8 -> 28.8, 4096 in chunks of 2048 59.7 -> 57.2.)
__host__ __device__ constexpr bool own_registers(int direct, bool f32) { return f32 && direct > 0; }
__host__ __device__ constexpr int f32_threads(int direct) { return direct ? 512 : kGemmThreads + 32 * convert_warps(direct); }

// bf16 roundings of fp32 operands, [batch, heads, len, head_dim] contiguous, written on the way (null: not wanted)
struct EstRounded {
  uint4 *q, *k;
  int q_len, k_len;
};

// The selection on rows that the epilogue has finished (EstGeom::direct): a chain of a microsecond per row, which runs under the
// next tiles' products, or, where a cluster of four has a single tile, on a warp per row.  As a kernel of its own it was a launch and a
// hand-over between two kernels more (1003 tokens: the prefill 26.2 -> 24.2 us; 128K tokens 773 -> 765 in short runs).
// Only the kernel of single CTAs with 128-column tiles of 16-bit operands does it: in the others the epilogue has no registers left for
// it (spills: 4096 tokens against 65536 51.9 -> 52.5 us a call although nothing was selected there), or, CTA pairs with their few
// steps per tile, no time (114688 tokens at stride 8 939 -> 967, 3590 tokens of a 16384-token chunk 34.5 -> 38.1).
// And only calls that select there take the kernel that can: the others' epilogue is the faster without that code (1003 tokens at
// stride 8 25.4 us a call with it, 24.5 without).
__host__ __device__ constexpr bool can_select(int direct, bool f32) { return direct == 1 && !f32; }
struct EstSelect {
  SelParams p;
  const float* thr_per_head;
  uint8_t* mask;
  int32_t *idx, *cnt;
};

struct EstNothing {};
template <bool kSelect>
using EstSelectIf = std::conditional_t<kSelect, EstSelect, EstNothing>;

struct EstGeom {
  int batch, hq, hkv;
  int S, d_chunks;             // K loop: S * d_chunks steps of 64 elements (fp32: of 32)
  int term_chunks;             // rows of bf16 terms of fp32 values: 64-column chunks per term (0: plain rows); see k_column
  int rows_total, cols_total;  // padded lengths / S
  int rows_valid, cols_valid;  // rows past rows_valid give zeros; causal: columns past cols_valid are hidden
  int rcs;                     // chunk_size / S
  int row_off;                 // (k_chunks - q_chunks) * rcs: global position of row 0
  int causal, left_blank;      // left_blank: columns left of the row's chunk are hidden (torch branch, un-padded K)
  int rbs, kb_total, qb_total;
  int n_mtiles, n_ntiles;
  int tile_n;                  // columns per tile: 256, or 128 when no row sees more than 128 columns
  int band;                    // attn_sums holds only the chunk's own key blocks (left_blank only): row stride bpc
  int bpc;                     // key blocks per chunk
  // Scratch layout: tile by tile, m_pitch tiles per row tile; a tile holds tile_n / rbs partial block sums and one (max, sum)
  // pair of each of its 128 rows, the rows of a block sum next to one another (the epilogue's lanes are rows, and
  // est_blocksum_kernel reads a block sum's 128 rows as one line).  Dense: every column tile.  Compact (left_blank: a row only ever
  // touches the tiles of its own chunk): the column tiles [tile_lo, tile_lo + m_pitch) of the row tile.
  int compact, m_pitch;
  // Lengths that are no multiple of the stride: the last stride group lacks the tokens of offset >= len % stride, which
  // count as zeros.  Two tensor maps of each operand: token offsets below the remainder go through one that has that group (and
  // no other offsets), the others through one of the whole groups (see load_tile).
  int q_rem, k_rem;
  int q_groups, k_groups;      // whole stride groups
  int row_cols;                // columns of the maps
  int head_dim;
  float scale_log2;
  FastDiv by_tiles, by_group, by_hq;     // tiles per head (of the kernel that runs), query heads per kv head, query heads
  // few tiles: the K loop of each is split over a cluster of `split` CTAs (1: persistent CTAs, a tile each at a time)
  int split;
  // CTA pairs: the two are query heads 2p, 2p + 1 of a kv group at the same rows (otherwise neighbouring row tiles of a head)
  int pair_heads;
  int direct;                  // the epilogue finishes the block sums: every row tile is computed, even one that sees nothing
  // Tile tables of est_setup_kernel computed on the host and carried in the kernel parameters when they are small
  // (tab_n = n_mtiles <= kTabTiles, e.g. 32 row tiles at 32K tokens, 64 at 128K): every kernel copies them into
  // shared memory and est_setup_kernel is not launched.  Layout: tile_lo[kTabTiles], tile_prefix[kTabTiles + 1],
  // pair_lo[kTabTiles / 2], pair_prefix[kTabTiles / 2 + 1].
  int tab_n;
  int tab[64 + 65 + 32 + 33];
};
constexpr int kTabTiles = 64;
constexpr int kTabInts = kTabTiles + (kTabTiles + 1) + kTabTiles / 2 + (kTabTiles / 2 + 1);
constexpr int kTabPrefix = kTabTiles, kTabPairLo = kTabPrefix + kTabTiles + 1, kTabPairPrefix = kTabPairLo + kTabTiles / 2;
static_assert(kTabInts == 64 + 65 + 32 + 33, "EstGeom::tab");

// Visible columns [lo, hi] of reshaped row i (empty when hi < lo).
// causal, torch branch (Xattention.py:191-225): columns [chunk_start, chunk_start + i_local], minus the
// K padding; when K is not padded the slice `[-0:]` at :201 hides everything left of the chunk too.
// causal, Triton (kernels.py:56): columns <= global position of the row.  non-causal: everything.
__host__ __device__ inline void row_bounds(const EstGeom& g, int i, int& lo, int& hi) {
  if (i >= g.rows_valid) { lo = 1; hi = 0; return; }
  if (!g.causal) { lo = 0; hi = g.cols_total - 1; return; }
  const int chunk_start = (i / g.rcs) * g.rcs + g.row_off;
  lo = g.left_blank ? chunk_start : 0;
  hi = g.row_off + i;
  if (hi > g.cols_valid - 1) hi = g.cols_valid - 1;
}

// Columns of both operands of step dc of a token.  Plain rows: one 64-column chunk after the other.  Rows of three bf16 terms
// [hi | mid | lo]: of one chunk after the other the three terms, three stages the MMA issuer treats as one.
__device__ __forceinline__ int k_column(const EstGeom& g, int dc) {
  if (g.term_chunks == 0) return dc * kTileK;
  const int c = dc / 3, term = dc - 3 * c;
  return (term * g.term_chunks + c) * kTileK;
}

// Loads a box of rows [row, row + box) of one token offset; `n_rows`: those that the map has of that offset.  A box without any
// of them is zeros, and is taken from past the columns of the tensor's first row: its own coordinates are out of bounds all the
// same, but name an address that can be far behind the tensor (3 tokens of 9 fp32 heads at stride 32: up to 290 KiB), and such
// loads have raised memory faults where nothing is mapped there.
template <bool kPair>
__device__ __forceinline__ void load_tile(const EstGeom& g, uint32_t dst, const CUtensorMap* m, uint32_t bar, int col, int offset, int row, int h,
                                          int b, int n_rows, uint32_t lead) {
  const bool in = row < n_rows;
  col = in ? col : g.row_cols;
  offset = in ? offset : 0;
  row = in ? row : 0;
  h = in ? h : 0;
  b = in ? b : 0;
  if constexpr (kPair) tma_load_5d_pair_lead(dst, m, bar, col, offset, row, h, b, lead);
  else tma_load_5d_lead(dst, m, bar, col, offset, row, h, b, lead);
}

// first column tile of a row tile's scratch, and the number of its tile (bh, mt, nt)
__host__ __device__ inline int scratch_tile0(const EstGeom& g, int nlo) { return g.compact ? nlo : 0; }
__device__ __forceinline__ size_t scratch_tile(const EstGeom& g, int bh, int mt, int nt, int nlo) {
  return (static_cast<size_t>(bh) * g.n_mtiles + mt) * g.m_pitch + nt - scratch_tile0(g, nlo);
}
// column-tile range of row tile mt: first tile and count (the formula of est_setup_kernel, also used by the host
// to size the compact scratch)
__host__ __device__ inline void row_tile_range(const EstGeom& g, int mt, int& first, int& count) {
  // lo(i) and hi(i) never decrease with i, so the tile's column range is [lo(first row), hi(last valid row)]
  const int i0 = mt * 128;
  int i1 = i0 + 128;
  if (i1 > g.rows_total) i1 = g.rows_total;
  if (i1 > g.rows_valid) i1 = g.rows_valid;
  int lo_min = 0, hi_max = -1;
  if (i1 > i0) {
    int lo, hi;
    row_bounds(g, i0, lo_min, hi);
    row_bounds(g, i1 - 1, lo, hi_max);
  }
  if (hi_max < lo_min) {
    first = 0;
    count = g.direct;
  } else {
    first = lo_min / g.tile_n;
    count = hi_max / g.tile_n - lo_min / g.tile_n + 1;
  }
}
// Whether row tile mt counts in the column-tile range of its pair (2p, 2p + 1), the union of the two: the second one does not
// if it sees nothing.  Its own range is then made up (the one tile that has its rows of the output zeroed, see EstGeom::direct)
// and would add column tiles that the first one does not see, for each of which the epilogue would write the first one's rows
// as zeros beside the sums of the right tile.  The first one's tile zeroes them as well.
__host__ __device__ inline bool counts_in_pair(const EstGeom& g, int mt) { return mt % 2 == 0 || mt * kTileM < g.rows_valid; }

// tile_lo[mt], tile_prefix[mt] (exclusive prefix of tile counts, n_mtiles+1 entries)
__global__ void est_setup_kernel(EstGeom g, int* __restrict__ tile_lo, int* __restrict__ tile_prefix,
                                 int* __restrict__ pair_lo, int* __restrict__ pair_prefix) {
  extern __shared__ int s_cnt[];                  // [n_mtiles] tile counts, then [n_mtiles] first tiles
  pdl_launch_dependents();
  pdl_wait();
  int* s_lo = s_cnt + g.n_mtiles;
  for (int mt = threadIdx.x; mt < g.n_mtiles; mt += blockDim.x) {
    row_tile_range(g, mt, s_lo[mt], s_cnt[mt]);
    tile_lo[mt] = s_lo[mt];
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    int acc = 0;
    for (int mt = 0; mt < g.n_mtiles; ++mt) {
      tile_prefix[mt] = acc;
      acc += s_cnt[mt];
    }
    tile_prefix[g.n_mtiles] = acc;
    // pairs of row tiles (2p, 2p+1) for the CTA-pair GEMM: the union of their column-tile ranges
    const int n_pairs = (g.n_mtiles + 1) / 2;
    acc = 0;
    for (int pm = 0; pm < n_pairs; ++pm) {
      int lo = 0x7fffffff, hi = -1;
      for (int mt = 2 * pm; mt < 2 * pm + 2 && mt < g.n_mtiles; ++mt)
        if (s_cnt[mt] > 0 && counts_in_pair(g, mt)) {
          lo = s_lo[mt] < lo ? s_lo[mt] : lo;
          hi = s_lo[mt] + s_cnt[mt] - 1 > hi ? s_lo[mt] + s_cnt[mt] - 1 : hi;
        }
      pair_lo[pm] = hi < 0 ? 0 : lo;
      pair_prefix[pm] = acc;
      acc += hi < 0 ? 0 : hi - lo + 1;
    }
    pair_prefix[n_pairs] = acc;
  }
}

// Tables from the kernel parameters (EstGeom::tab) copied into shared memory by the whole CTA; the caller
// synchronises the CTA before the first use.
__device__ __forceinline__ void load_tables(const EstGeom& g, int* s_tab) {
  for (int i = threadIdx.x; i < kTabInts; i += blockDim.x) s_tab[i] = g.tab[i];
}

// Tile number -> (batch*head, row-tile group, column tile).  With `interleave` > 1 (the query heads per kv head)
// the heads of a kv group take the same (row, column) tile one after the other, so that the K tile they share is
// read from DRAM once and found in L2 by the other heads: it matters when the kernel streams its operands from
// HBM (128-column tiles), where K otherwise came from DRAM about twice.
__device__ __forceinline__ void decode_tile(const EstGeom& g, int n_groups, const int* __restrict__ tile_lo,
                                            const int* __restrict__ tile_prefix, int tile, int& bh, int& mt, int& nt,
                                            bool interleave = false) {
  int rem, hg = 0;
  if (interleave) tile = fast_div(tile, g.by_group, hg);     // hg: head inside its kv group
  bh = fast_div(tile, g.by_tiles, rem);
  if (interleave) bh = bh * static_cast<int>(g.by_group.d) + hg;
  int lo = 0, hi = n_groups;     // find mt with prefix[mt] <= rem < prefix[mt+1]
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (tile_prefix[mid] <= rem) lo = mid; else hi = mid;
  }
  mt = lo;
  nt = tile_lo[mt] + rem - tile_prefix[mt];
}

// Epilogue of one accumulator tile for one row (thread): softmax statistics and un-normalised block sums of the
// tile's visible columns [clo, chi].  Two passes over the row in tensor memory (maximum, then exp2 and sums over
// groups of RBS columns), the load of the next 32 columns in flight while the current ones are processed; chunks
// that every lane of the warp sees completely skip the per-element range test.  `part`: this row's first partial sum, the
// next key block's is kTileM floats on (a warp stores 128 contiguous bytes).  `release` is called once all
// tensor-memory reads of the tile are done.
template <int RBS, typename Release>
__device__ __forceinline__ void est_epilogue_row(const EstGeom& g, uint32_t taddr, int n_chunks, int clo, int chi,
                                                 bool write, float* __restrict__ part, float2* __restrict__ mslot,
                                                 Release release) {
  // columns hidden from this row become -inf, in chunks that some row of the warp sees only in part
  auto hide = [&](uint32_t (&v)[32], int c8) {
    if (!__all_sync(0xffffffffu, clo <= c8 * 32 && chi >= c8 * 32 + 31)) {
#pragma unroll
      for (int k = 0; k < 32; ++k) v[k] = c8 * 32 + k >= clo && c8 * 32 + k <= chi ? v[k] : 0xff800000u;
    }
  };
  // pass 1: row maximum over the visible columns
  float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
  {
    auto max_chunk = [&](uint32_t (&v)[32], int c8) {
      hide(v, c8);
#pragma unroll
      for (int k = 0; k < 16; ++k) mx4[k & 3] = max3(mx4[k & 3], __uint_as_float(v[2 * k]), __uint_as_float(v[2 * k + 1]));
    };
    uint32_t va[32], vb[32];
    tmem_ld32(taddr, va);
#pragma unroll 1
    for (int c8 = 0; c8 < n_chunks; c8 += 2) {
      tc_wait_ld();
      tmem_ld32(taddr + (c8 + 1) * 32, vb);
      max_chunk(va, c8);
      tc_wait_ld();
      if (c8 + 2 < n_chunks) tmem_ld32(taddr + (c8 + 2) * 32, va);
      max_chunk(vb, c8 + 1);
    }
  }
  const float m_scaled = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3])) * g.scale_log2;     // scale > 0
  // pass 2: exp2 and sums over groups of RBS columns
  const float m_ref = m_scaled == -INFINITY ? 0.f : m_scaled;
  const unsigned long long scale2 = pack_f32x2(g.scale_log2, g.scale_log2), nm2 = pack_f32x2(-m_ref, -m_ref);
  float tile_sum = 0.f;
  {
    auto sum_chunk = [&](uint32_t (&v)[32], int c8) {
      hide(v, c8);
      float gs[32 / RBS];
#pragma unroll
      for (int q = 0; q < 32 / RBS; ++q) {
        unsigned long long s2 = 0ull;
#pragma unroll
        for (int k = q * RBS / 2; k < (q + 1) * RBS / 2; ++k) {
          float y0, y1;
          unpack_f32x2(fma_f32x2(pack_f32x2(__uint_as_float(v[2 * k]), __uint_as_float(v[2 * k + 1])), scale2, nm2), y0, y1);
          s2 = add_f32x2(s2, pack_f32x2(fast_exp2(y0), fast_exp2(y1)));
        }
        float a, b;
        unpack_f32x2(s2, a, b);
        gs[q] = a + b;
      }
#pragma unroll
      for (int q = 0; q < 32 / RBS; ++q) tile_sum += gs[q];
      if (write) {
#pragma unroll
        for (int q = 0; q < 32 / RBS; ++q) part[(c8 * (32 / RBS) + q) * kTileM] = gs[q];
      }
    };
    uint32_t va[32], vb[32];
    tmem_ld32(taddr, va);
#pragma unroll 1
    for (int c8 = 0; c8 < n_chunks; c8 += 2) {
      tc_wait_ld();
      tmem_ld32(taddr + (c8 + 1) * 32, vb);
      sum_chunk(va, c8);
      tc_wait_ld();
      if (c8 + 2 < n_chunks) tmem_ld32(taddr + (c8 + 2) * 32, va);
      else release();                                   // the tile's last load has completed
      sum_chunk(vb, c8 + 1);
    }
  }
  if (write) *mslot = make_float2(m_scaled, tile_sum);
}

// Epilogue for geometries in which a reshaped row sees a single column tile (the torch branch with chunks of 128 or 256
// reshaped rows, e.g. 128K or 64K tokens at stride 16; prompts of that many columns altogether): the tile's row maximum and
// row sum ARE the row's, so the normalised block sums are finished here -- exp2 against the row maximum, sums over groups of
// RBS columns kept in registers, division by the row sum, and the sum over the RBS rows of a query block taken across lanes
// -- and written to the block sums directly.  Neither the per-row scratch nor the two kernels that would read it are needed.
// `out`: the query block's row of out_cols sums, the tile's first one at col0; the others are zero.
//
// The row's scores come in halves of 128 columns (`load(half, v)`; chunks of 32 columns from `nvis` on are hidden from the
// whole warp), each in registers as a whole: one tensor-memory round trip for 128 columns, and the lower half once more for
// 256.  The block sums of the RBS rows of a query block are added by halves: a lane gives away half of its sums and receives
// the other lane's part of the half it keeps, 14 shuffles for 8 rows of 16 sums instead of 48.
template <int RBS, int kHalves, typename Load>
__device__ __forceinline__ void est_epilogue_row_direct(const EstGeom& g, Load load, int nvis, int clo, int chi,
                                                        float* __restrict__ out, int col0, int out_cols, bool write, int lane) {
  constexpr int kBlocks = kHalves * 128 / RBS, kPer = 32 / RBS;
  uint32_t v[4][32];
  float mx8[8];
#pragma unroll
  for (int q = 0; q < 8; ++q) mx8[q] = -INFINITY;
  auto hide = [&](int half) {
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const int c0 = half * 128 + c * 32;
      if (half * 4 + c < nvis && !__all_sync(0xffffffffu, clo <= c0 && chi >= c0 + 31)) {
#pragma unroll
        for (int k = 0; k < 32; ++k) v[c][k] = c0 + k >= clo && c0 + k <= chi ? v[c][k] : 0xff800000u;
      }
    }
  };
#pragma unroll
  for (int half = 0; half < kHalves; ++half) {
    if (half * 4 >= nvis && half > 0) continue;
    load(half, v);
    hide(half);
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      if (half * 4 + c >= nvis) continue;
#pragma unroll
      for (int k = 0; k < 16; ++k)
        mx8[k & 7] = max3(mx8[k & 7], __uint_as_float(v[c][2 * k]), __uint_as_float(v[c][2 * k + 1]));
    }
  }
  const float mx = fmaxf(max3(mx8[0], mx8[1], mx8[2]), max3(max3(mx8[3], mx8[4], mx8[5]), mx8[6], mx8[7]));
  const float m = mx == -INFINITY ? 0.f : mx * g.scale_log2;           // scale > 0
  const unsigned long long scale2 = pack_f32x2(g.scale_log2, g.scale_log2), nm2 = pack_f32x2(-m, -m);
  float blk[kBlocks];
  float row_sum = 0.f;
  // the upper half is still in registers; the lower one of two is loaded again
#pragma unroll
  for (int half = kHalves - 1; half >= 0; --half) {
    if (kHalves == 2 && half == 0 && nvis > 4) {
      load(0, v);
      hide(0);
    }
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const int b0 = (half * 4 + c) * kPer;
#pragma unroll
      for (int q = 0; q < kPer; ++q) blk[b0 + q] = 0.f;
      if (half * 4 + c >= nvis) continue;
#pragma unroll
      for (int q = 0; q < kPer; ++q) {
        unsigned long long s2 = 0ull;
#pragma unroll
        for (int k = q * RBS / 2; k < (q + 1) * RBS / 2; ++k) {
          float y0, y1;
          unpack_f32x2(fma_f32x2(pack_f32x2(__uint_as_float(v[c][2 * k]), __uint_as_float(v[c][2 * k + 1])), scale2, nm2), y0, y1);
          s2 = add_f32x2(s2, pack_f32x2(fast_exp2(y0), fast_exp2(y1)));
        }
        float a, b;
        unpack_f32x2(s2, a, b);
        blk[b0 + q] = a + b;
        row_sum += a + b;
      }
    }
  }
  // normalise (a row that sees nothing contributes nothing), then add the RBS rows of the query block, RBS lanes
  const float inv = row_sum > 0.f ? 1.f / row_sum : 0.f;
#pragma unroll
  for (int q = 0; q < kBlocks; ++q) blk[q] *= inv;
  int n = kBlocks, base = 0;
#pragma unroll
  for (int o = 1; o < RBS; o <<= 1) {
    if (n > 1) {
      n >>= 1;
      const bool upper = (lane & o) != 0;
      if (upper) base += n;
#pragma unroll
      for (int j = 0; j < kBlocks / 2; ++j)
        if (j < n) blk[j] = (upper ? blk[j + n] : blk[j]) + __shfl_xor_sync(0xffffffffu, upper ? blk[j] : blk[j + n], o);
    } else {
      write = write && (lane & o) == 0;                                // (more lanes than sums)
      blk[0] += __shfl_xor_sync(0xffffffffu, blk[0], o);
    }
  }
  if (!write) return;
  constexpr int kLeft = kBlocks > RBS ? kBlocks / RBS : 1;
#pragma unroll
  for (int q = 0; q < kLeft; ++q)
    if (col0 + base + q < out_cols) out[col0 + base + q] = blk[q];
  // (dense rows of more blocks than the tile holds)
  constexpr int kWriters = kBlocks > RBS ? RBS : kBlocks;
  const int outside = out_cols - (out_cols - col0 < kBlocks ? out_cols - col0 : kBlocks);
#pragma unroll 1
  for (int c = base / kLeft; c < outside; c += kWriters) out[c < col0 ? c : c + kBlocks] = 0.f;
}

// Selects query blocks [qb0, qb0 + n) of a head, whose sums this warp (or, behind a barrier, its CTA) has written: every
// `step`-th of them from the `first` on.
__device__ __forceinline__ void est_select_rows(const EstGeom& g, const EstSelect& sel, const float* sums, int bh, int qb0, int n, int first,
                                                int step, int lane) {
  __syncwarp();
#pragma unroll 1
  for (int r = first; r < n && qb0 + r < g.qb_total; r += step)
    select_row<1>(sums, sel.p, sel.thr_per_head, sel.mask, sel.idx, sel.cnt, bh * g.qb_total + qb0 + r, lane);
}

// Eight fp32 values, in pairs: the next term of each, the rounding of what the terms before leave.
__device__ __forceinline__ uint4 next_term(unsigned long long (&v)[4]) {
  uint32_t w[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    float x, y;
    unpack_f32x2(v[k], x, y);
    const __nv_bfloat162 p = __floats2bfloat162_rn(x, y);
    w[k] = *reinterpret_cast<const uint32_t*>(&p);
    v[k] = fma_f32x2(pack_f32x2(__low2float(p), __high2float(p)), pack_f32x2(-1.f, -1.f), v[k]);
  }
  return make_uint4(w[0], w[1], w[2], w[3]);
}

// kDirect: 128-column halves per row of the epilogue above, 0: the general one
// kF32: fp32 operands.  x = hi + mid + lo in bf16 (each the rounding of what the ones before it leave), and the six products
// of terms that reach 2^-24 of the first: hh; hm, mh, mm; hl, lh.  The split happens here, between the loads and the MMAs:
// more warps take the fp32 units from shared memory and write the terms to shared memory, half of a 64-column stage while the
// MMAs read the other.  Terms written to HBM first cost 10 bytes per element, and the GEMM then found HBM busy with writing
// them back (32 heads of 4096 tokens, chunks of 2048: split 56 us + GEMM 46 -> 44; the prefill, whose attention phase takes the
// bf16 roundings written here, 151 -> 114 us, 2 us of them for the proxy fence of every unit).  Bound by the latency of a
// converter's step (waits, shared-memory traffic next to the MMAs', three dependent roundings); with loads alone it runs in 30
// us.  Sixteen converter warps, or eight beside an epilogue with registers of its own (own_registers).
// kSelect: and selects on its rows (can_select)
template <int RBS, int kDirect, bool kF32, bool kSelect>
__global__ void __launch_bounds__(kF32 ? f32_threads(kDirect) : kGemmThreads, 1)
est_gemm_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                const __grid_constant__ CUtensorMap tmQt, const __grid_constant__ CUtensorMap tmKt, const EstGeom g,
                const int* tile_lo, const int* tile_prefix, float* __restrict__ partial,
                float2* __restrict__ mtile, float* sums, const uint32_t idesc, const EstRounded rounded, const EstSelectIf<kSelect> sel, int* status) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ int s_tab[kTabInts];
  if (g.tab_n) {                                  // (made visible by the __syncthreads() that ends the prologue)
    load_tables(g, s_tab);
    tile_lo = s_tab;
    tile_prefix = s_tab + kTabPrefix;
  }
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  // 128-column tiles (every operand tile is used once: the kernel streams Q and K from HBM) take six 32 KiB
  // stages, 256-column tiles four 48 KiB ones: 192 KiB in flight either way
  // (fp32: three stages' space for the terms, the rest the ring of units)
  const int stage_bytes = kABytes + g.tile_n * kTileK * 2;
  const int n_stages = kF32 ? (kF32Smem - 3 * stage_bytes) / kF32Unit : (g.tile_n == 128 ? kMaxStages : kStages);
  constexpr int kBars = kF32 ? kMaxUnits : kMaxStages;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + (kF32 ? kF32Smem : kStages * kStageBytes));
  const uint32_t full0 = smem_u32(bars);                       // [kBars]
  const uint32_t empty0 = smem_u32(bars + kBars);              // [kBars]
  const uint32_t tfull0 = smem_u32(bars + 2 * kBars);          // [2]
  const uint32_t tempty0 = smem_u32(bars + 2 * kBars + 2);     // [2]
  const uint32_t terms_full0 = smem_u32(bars + 2 * kBars + 4); // [2] (fp32) terms of 32 columns written / read
  const uint32_t terms_empty0 = smem_u32(bars + 2 * kBars + 6);// [2]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * kBars + 8);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);     // (uniform for the compiler too)
  const int lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kBars; ++s) {
      mbar_init(full0 + 8 * s, 1);
      mbar_init(empty0 + 8 * s, kF32 ? convert_warps(kDirect) : 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(tfull0 + 8 * a, 1);
      mbar_init(tempty0 + 8 * a, 4);
      mbar_init(terms_full0 + 8 * a, convert_warps(kDirect));
      mbar_init(terms_empty0 + 8 * a, 1);
    }
    *abort_flag = 0;
    fence_mbar_init();
    tma_prefetch_desc(&tmQ);
    tma_prefetch_desc(&tmK);
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(tmem_slot), 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  pdl_launch_dependents();
  pdl_wait();                       // up to here nothing was touched that an earlier kernel writes
  const uint32_t tmem_base = *tmem_slot;

  const int tiles_per_head = tile_prefix[g.n_mtiles];
  const int total_tiles = tiles_per_head * g.batch * g.hq;
  // this CTA's tiles and its part of their K loop
  const int split = g.split, rank = split > 1 ? static_cast<int>(cluster_ctarank()) : 0;
  const int tile0 = blockIdx.x / split, tile_step = gridDim.x / split;
  const int k_steps = g.S * g.d_chunks, ks0 = k_steps * rank / split, ks1 = k_steps * (rank + 1) / split;
  const bool interleave = g.tile_n == 128 && g.hq > g.hkv;      // streaming case only: see decode_tile

  auto load_role = [&]() {
    // ------------------------------------------------------------ TMA producer (converged warp, one thread issues)
    {
      const uint32_t lead = elect_one() ? 1u : 0u;
      int s = 0;
      uint32_t ph = 0;
      for (int tile = tile0; tile < total_tiles && !*abort_flag; tile += tile_step) {
        int bh, mt, nt;
        decode_tile(g, g.n_mtiles, tile_lo, tile_prefix, tile, bh, mt, nt, interleave);
        int h, hg_;
        const int b = fast_div(bh, g.by_hq, h), hkv = fast_div(h, g.by_group, hg_);
        int t = ks0 / g.d_chunks, dc = ks0 - t * g.d_chunks;
        for (int ks = ks0; ks < ks1; ++ks) {
          const bool qt = g.S - 1 - t < g.q_rem, kt = t < g.k_rem;
          if constexpr (kF32) {
            bool ok = true;
            for (int n = -kTileM; n < g.tile_n && ok; n += kTileM) {         // A, then 128 rows of B at a time
              ok = __all_sync(0xffffffffu, mbar_wait(empty0 + 8 * s, ph ^ 1, abort_flag));
              if (!ok) break;
              const uint32_t dst = smem_u32(smem + 3 * stage_bytes + s * kF32Unit);
              mbar_expect_tx_lead(full0 + 8 * s, kF32Unit, lead);
              if (n < 0)
                load_tile<false>(g, dst, qt ? &tmQt : &tmQ, full0 + 8 * s, dc * kF32Cols, g.S - 1 - t, mt * kTileM, h, b, g.q_groups + qt, lead);
              else
                load_tile<false>(g, dst, kt ? &tmKt : &tmK, full0 + 8 * s, dc * kF32Cols, t, nt * g.tile_n + n, hkv, b, g.k_groups + kt, lead);
              if (++s == n_stages) { s = 0; ph ^= 1; }
            }
            if (!ok) break;
          } else {
            if (!__all_sync(0xffffffffu, mbar_wait(empty0 + 8 * s, ph ^ 1, abort_flag))) break;
            const uint32_t dstA = smem_u32(smem + s * stage_bytes);
            mbar_expect_tx_lead(full0 + 8 * s, stage_bytes, lead);
            load_tile<false>(g, dstA, qt ? &tmQt : &tmQ, full0 + 8 * s, dc * kTileK, g.S - 1 - t, mt * kTileM, h, b, g.q_groups + qt, lead);
            load_tile<false>(g, dstA + kABytes, kt ? &tmKt : &tmK, full0 + 8 * s, dc * kTileK, t, nt * g.tile_n, hkv, b, g.k_groups + kt, lead);
            if (++s == n_stages) { s = 0; ph ^= 1; }
          }
          if (++dc == g.d_chunks) { dc = 0; ++t; }
        }
      }
    }
    if (split > 1) {
      cluster_sync_all();
      cluster_sync_all();
    }
  };
  auto mma_role = [&]() {
    // ------------------------------------------------------------ MMA issuer (converged warp, one thread issues: see mma_ss_lead)
    {
      const uint32_t lead = elect_one() ? 1u : 0u;
      auto wait = [&](uint32_t bar, uint32_t ph) { return __all_sync(0xffffffffu, mbar_wait(bar, ph, abort_flag)); };
      int st = 0;
      uint32_t ph = 0, local_tile = 0;
      const uint64_t a_desc0 = smem_desc_sw128(smem_u32(smem), 16, 1024);
      const uint64_t b_desc0 = smem_desc_sw128(smem_u32(smem) + kABytes, 16, 1024);
      for (int tile = tile0; tile < total_tiles && !*abort_flag; tile += tile_step, ++local_tile) {
        const uint32_t acc = local_tile & 1;
        const uint32_t acc_ph = (local_tile >> 1) & 1;
        if (!wait(tempty0 + 8 * acc, acc_ph ^ 1)) break;
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + acc * kTileN;
        bool ok = true;
        for (int ks = ks0; ks < ks1; ++ks) {
          if (!wait(kF32 ? terms_full0 + 8 * st : full0 + 8 * st, ph)) { ok = false; break; }
          tc_fence_after();
          // D += A of stage sa * B of stage sb, 16-column steps [k0, k1); descriptors differ from the stage-0 ones only in the
          // start-address field (units of 16 bytes)
          auto product = [&](int sa, int sb, int k0, int n, uint32_t accumulate) {
            const uint64_t a_desc = a_desc0 + static_cast<uint64_t>(sa * (stage_bytes >> 4) + 2 * k0);
            const uint64_t b_desc = b_desc0 + static_cast<uint64_t>(sb * (stage_bytes >> 4) + 2 * k0);
#pragma unroll
            for (int k = 0; k < n; ++k) mma_ss_lead(d_tmem, a_desc + k * 2, b_desc + k * 2, idesc, k > 0 ? 1u : accumulate, lead);
          };
          if constexpr (kF32) {
            const int k0 = st * (kF32Cols / 16);
            product(0, 0, k0, kF32Cols / 16, ks > ks0 ? 1u : 0u);
            product(0, 1, k0, kF32Cols / 16, 1u);
            product(1, 0, k0, kF32Cols / 16, 1u);
            product(1, 1, k0, kF32Cols / 16, 1u);
            product(0, 2, k0, kF32Cols / 16, 1u);
            product(2, 0, k0, kF32Cols / 16, 1u);
            mma_commit_lead(terms_empty0 + 8 * st, lead);
            if (++st == 2) { st = 0; ph ^= 1; }
          } else {
            product(st, st, 0, kTileK / 16, ks > ks0 ? 1u : 0u);
            mma_commit_lead(empty0 + 8 * st, lead);       // stage reusable once these MMAs have read it
            if (++st == n_stages) { st = 0; ph ^= 1; }
          }
        }
        if (!ok) break;
        mma_commit_lead(tfull0 + 8 * acc, lead);          // accumulator complete
      }
    }
    if (split > 1) {
      cluster_sync_all();
      cluster_sync_all();
    }
  };
  constexpr int kFirstConverter = own_registers(kDirect, kF32) ? 8 : kGemmThreads / 32;
  auto convert_role = [&]() {
    if constexpr (kF32) {
    // ------------------------------------------------------------ converters (fp32): some rows of each unit per warp
    // A lane takes eight columns (two 16-byte chunks) of one row of each group of eight.  Rows p and p ^ 5 next to one another:
    // neither the fp32 reads (chunks 2 col, 2 col + 1 of a swizzled row) nor the term writes (chunk col of a half) of a
    // quarter-warp then share a bank.
    constexpr int kGroups = kTileM / 8 / convert_warps(kDirect);
    const int col = lane & 3, r7 = (lane >> 3) ^ ((lane >> 2 & 1) * 5), row0 = (warp - kFirstConverter) * 8 * kGroups + r7;
    const uint32_t src0 = smem_u32(smem) + 3 * stage_bytes + row0 * 128, ch0 = ((2 * col) ^ r7) * 16, ch1 = ((2 * col + 1) ^ r7) * 16;
    const int row_vecs = g.head_dim / 8;
    int s = 0, half = 0;
    uint32_t ph = 0, half_ph = 0;
    bool ok = true;
    auto wait = [&](uint32_t bar, uint32_t parity) { return __all_sync(0xffffffffu, mbar_wait(bar, parity, abort_flag)); };
    for (int tile = tile0; tile < total_tiles && ok; tile += tile_step) {
      int bh, mt, nt, h, hg;
      decode_tile(g, g.n_mtiles, tile_lo, tile_prefix, tile, bh, mt, nt, interleave);
      const int b = fast_div(bh, g.by_hq, h), hkv = fast_div(h, g.by_group, hg);
      // the roundings are written by the first tile of a row tile, and by the first one that has the column tile
      uint4* q_out = nt == tile_lo[mt] ? rounded.q : nullptr;
      uint4* k_out = hg == 0 && (mt == 0 || nt >= tile_lo[mt - 1] + tile_prefix[mt] - tile_prefix[mt - 1]) ? rounded.k : nullptr;
      if (q_out) q_out += static_cast<size_t>(bh) * rounded.q_len * row_vecs + col;
      if (k_out) k_out += static_cast<size_t>(b * g.hkv + hkv) * rounded.k_len * row_vecs + col;
      int t = ks0 / g.d_chunks, dc = ks0 - t * g.d_chunks;
#pragma unroll 1
      for (int ks = ks0; ks < ks1 && ok; ++ks) {
        if (!wait(terms_empty0 + 8 * half, half_ph ^ 1)) { ok = false; break; }
#pragma unroll 1
        for (int n = -kTileM; n < g.tile_n; n += kTileM) {                   // A, then 128 rows of B at a time
          if (!wait(full0 + 8 * s, ph)) { ok = false; break; }
          unsigned long long v[kGroups][4];
#pragma unroll
          for (int i = 0; i < kGroups; ++i) {
            const uint32_t src = src0 + s * kF32Unit + i * 8 * 128;
            ld_shared_2b64(src + ch0, v[i][0], v[i][1]);
            ld_shared_2b64(src + ch1, v[i][2], v[i][3]);
          }
          uint4 term[3][kGroups];                        // (all groups term by term: their chains of conversions overlap)
#pragma unroll
          for (int e = 0; e < 3; ++e)
#pragma unroll
            for (int i = 0; i < kGroups; ++i) term[e][i] = next_term(v[i]);
          const uint32_t dst = smem_u32(smem) + (n < 0 ? 0 : kABytes + n * 128) + row0 * 128 + (((4 * half + col) ^ r7) * 16);
          uint4* out = n < 0 ? q_out : k_out;
          const int out_len = out ? (n < 0 ? rounded.q_len : rounded.k_len) : 0;
          const int token = ((n < 0 ? mt * kTileM : nt * g.tile_n + n) + row0) * g.S + (n < 0 ? g.S - 1 - t : t);
#pragma unroll
          for (int i = 0; i < kGroups; ++i)
#pragma unroll
            for (int e = 0; e < 3; ++e) st_shared_v4(dst + i * 8 * 128 + e * stage_bytes, term[e][i]);
          // The unit goes back to TMA, which writes through the async proxy: a proxy fence of every lane orders its reads before
          // that.  (Without one, an arrival right behind the reads gave wrong terms.)  It orders the lane's stores of terms before
          // the MMAs' reads, too, the last unit's those of the whole step.
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) mbar_arrive(empty0 + 8 * s);
          if (++s == n_stages) { s = 0; ph ^= 1; }
#pragma unroll
          for (int i = 0; i < kGroups; ++i)
            if (token + i * 8 * g.S < out_len) out[static_cast<size_t>(token + i * 8 * g.S) * row_vecs + dc * 4] = term[0][i];
        }
        if (!ok) break;
        if (lane == 0) mbar_arrive(terms_full0 + 8 * half);
        if (++half == 2) { half = 0; half_ph ^= 1; }
        if (++dc == g.d_chunks) { dc = 0; ++t; }
      }
    }
    if (split > 1) {
      cluster_sync_all();
      cluster_sync_all();
    }
    }
  };
  auto epilogue_role = [&]() {
    // ------------------------------------------------------------ epilogue (4 warps, thread = tile row)
    const int quad = warp & 3;                  // TMEM lane quarter this warp may access
    const int r = quad * 32 + lane;
    const int kGroups = g.tile_n / RBS;         // key blocks per tile
    const int n_chunks = g.tile_n / 32;
    uint32_t local_tile = 0;
    for (int tile = tile0; tile < total_tiles; tile += tile_step, ++local_tile) {
      int bh, mt, nt;
      decode_tile(g, g.n_mtiles, tile_lo, tile_prefix, tile, bh, mt, nt, interleave);
      const uint32_t acc = local_tile & 1;
      const uint32_t acc_ph = (local_tile >> 1) & 1;
      const int i = mt * kTileM + r;
      int lo, hi;
      row_bounds(g, i, lo, hi);
      const int n0 = nt * g.tile_n;
      const int clo = lo - n0 > 0 ? lo - n0 : 0;
      const int chi = hi - n0 < g.tile_n - 1 ? hi - n0 : g.tile_n - 1;
      // warp-uniform: the tensor-memory loads below are warp-collective
      const bool ok = __all_sync(0xffffffffu, mbar_wait(tfull0 + 8 * acc, acc_ph, abort_flag));
      if (!ok && split == 1) break;                   // (a cluster's barriers are passed in any case)
      tc_fence_after();
      const uint32_t taddr = tmem_base + acc * kTileN + (static_cast<uint32_t>(quad * 32) << 16);
      // 32-column chunks that some row of the warp sees
      const int nvis = min((__reduce_max_sync(0xffffffffu, chi >= clo ? chi : -1) + 32) >> 5, n_chunks);
      // of this warp's quarter of the rows: the chunk in the parts that the other CTAs of the cluster sent
      const int own = 4 / split;                      // quarters a CTA finishes
      auto add_parts = [&](uint32_t (&v)[32], int c) {
        for (int src = 0; src < split - 1; ++src) {
          const uint8_t* from = smem + (src * own + quad % own) * g.tile_n * 128 + c * 8 * 512 + lane * 16;
#pragma unroll
          for (int q4 = 0; q4 < 8; ++q4) {
            const float4 x = *reinterpret_cast<const float4*>(from + q4 * 512);
            v[4 * q4] = __float_as_uint(__uint_as_float(v[4 * q4]) + x.x);
            v[4 * q4 + 1] = __float_as_uint(__uint_as_float(v[4 * q4 + 1]) + x.y);
            v[4 * q4 + 2] = __float_as_uint(__uint_as_float(v[4 * q4 + 2]) + x.z);
            v[4 * q4 + 3] = __float_as_uint(__uint_as_float(v[4 * q4 + 3]) + x.w);
          }
        }
      };
      if (split > 1) {
        // The cluster's accumulators are added up, every CTA finishing 128 / split rows: the others' parts of them come
        // through its shared memory ([source][32-row quarter][4 columns][lane] of 16 bytes; the operand stages, which no CTA
        // reads any more).  (The loader and issuer warps keep the barriers company below.)
        const int dest = quad / own;                  // the CTA that finishes this warp's rows
        cluster_sync_all();
        if (dest != rank) {
          const int slot = rank < dest ? rank : rank - 1;
          const uint32_t base = mapa_shared(smem_u32(smem) + (slot * own + quad % own) * g.tile_n * 128 + lane * 16, dest);
#pragma unroll 1
          for (int c = 0; c < nvis; ++c) {
            uint32_t v[32];
            tmem_ld32(taddr + c * 32, v);
            tc_wait_ld();
#pragma unroll
            for (int q4 = 0; q4 < 8; ++q4) st_shared_cluster_v4(base + (c * 8 + q4) * 512, v[4 * q4], v[4 * q4 + 1], v[4 * q4 + 2], v[4 * q4 + 3]);
          }
        }
        cluster_sync_all();
        if (dest != rank || !ok) break;
        if (kDirect == 0) {
#pragma unroll 1
          for (int c = 0; c < nvis; ++c) {
            uint32_t v[32];
            tmem_ld32(taddr + c * 32, v);
            tc_wait_ld();
            add_parts(v, c);
            tmem_st32(taddr + c * 32, v);
          }
          tc_wait_st();
        }
      }
      auto release = [&]() {
        // all TMEM reads of this accumulator are done: hand it back to the MMA thread
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(tempty0 + 8 * acc);
      };
      if constexpr (kDirect > 0) {
        // the query block of this row, and its first row's lane as the writer (RBS divides 32)
        const int qb = i / RBS;
        const int out_cols = g.band ? g.bpc : g.kb_total, col0 = g.band ? 0 : nt * kGroups;
        // (the accumulator goes back to the MMA thread with the last read: the second one of the lower half, if it is read again)
        int reads = kDirect == 2 && nvis > 4 ? 3 : 1;
        auto load = [&](int half, uint32_t (&v)[4][32]) {
#pragma unroll
          for (int c = 0; c < 4; ++c) tmem_ld32(taddr + half * 128 + c * 32, v[c]);
          tc_wait_ld();
          if (--reads == 0) release();
          if (split > 1) {
#pragma unroll
            for (int c = 0; c < 4; ++c)
              if (half * 4 + c < nvis) add_parts(v[c], half * 4 + c);
          }
        };
        est_epilogue_row_direct<RBS, kDirect>(g, load, nvis, clo, chi,
                                              sums + (static_cast<size_t>(bh) * g.qb_total + (qb < g.qb_total ? qb : 0)) * out_cols, col0, out_cols,
                                              qb < g.qb_total, lane);
        if constexpr (kSelect) {
          if (split == 1) est_select_rows(g, sel, sums, bh, (mt * kTileM + quad * 32) / RBS, 32 / RBS, 0, 1, lane);
        }
      } else {
        const size_t tile_at = scratch_tile(g, bh, mt, nt, tile_lo[mt]) * kTileM;
        est_epilogue_row<RBS>(g, taddr, n_chunks, clo, chi, true, partial + tile_at * kGroups + r, mtile + tile_at + r, release);
      }
    }
  };

  if constexpr (own_registers(kDirect, kF32)) {
    constexpr int kRegEpilogue = 192, kRegLoadMma = 64;
    static_assert(4 * kRegEpilogue + 4 * kRegLoadMma + 8 * 128 <= 16 * 128, "register budget of the roles");
    if (warp < 4) {
      reg_set_from<kRegLoadMma, 128>();
      if (warp == 0) {
        load_role();
      } else if (warp == 1) {
        mma_role();
      } else if (split > 1) {
        cluster_sync_all();
        cluster_sync_all();
      }
    } else if (warp < 8) {
      reg_set_from<kRegEpilogue, 128>();
      epilogue_role();
    } else {
      convert_role();
    }
  } else if (warp == 0) {
    load_role();
  } else if (warp == 1) {
    mma_role();
  } else if (kF32 && warp >= kFirstConverter) {
    convert_role();
  } else {
    epilogue_role();
  }

  // ---------------------------------------------------------------- teardown
  tc_fence_before();
  __syncthreads();
  if (*abort_flag) {
    // give copies and MMAs still in flight time to land before shared/tensor memory is released
    const long long t0 = clock64();
    while (clock64() - t0 < 2000000) { __nanosleep(1000); }
    if (threadIdx.x == 0 && status) atomicExch(status, static_cast<int>(kDevWaitTimeout));
    if constexpr (kSelect)
      for (int tile = tile0; tile < total_tiles; tile += tile_step) {
        int bh, mt, nt;
        decode_tile(g, g.n_mtiles, tile_lo, tile_prefix, tile, bh, mt, nt, interleave);
        forget_rows(sel.p, sel.mask, sel.cnt, bh, (mt * kTileM + rank * (kTileM / split)) / RBS, kTileM / split / RBS);
      }
    __syncthreads();
  } else if constexpr (kSelect) {
    if (split > 1) {
      // a cluster's CTA has finished 128 / split rows, few query blocks: a warp each
      int bh, mt, nt;
      decode_tile(g, g.n_mtiles, tile_lo, tile_prefix, tile0, bh, mt, nt, interleave);
      est_select_rows(g, sel, sums, bh, (mt * kTileM + rank * (kTileM / split)) / RBS, kTileM / split / RBS, warp,
                      static_cast<int>(blockDim.x >> 5), lane);
    }
  }
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

// The same GEMM on CTA PAIRS (thread-block clusters of 2, tcgen05 cta_group::2): a pair computes a 256x256 tile.
// Each CTA loads its own 128 rows of A and HALF of the tile's 256 columns of B (32 KiB per K step instead of 48),
// the even CTA issues 256x256x16 MMAs that read both CTAs' shared memory, and each CTA finds the accumulator of
// its own 128 rows in its own tensor memory, where its four epilogue warps work exactly as in the single-CTA
// kernel.  The single-CTA kernel is bound by operand bytes in flight per SM (L2 latency x shared-memory
// capacity); the pair moves a third fewer bytes per FLOP and has six 32 KiB stages in flight.
// The pair's rows are the same 128 of two query heads that share a kv head, if there are such (pair_heads): both see the
// same columns, so that a tile of which they see only the first 128 (every other one on the diagonal) is computed 128
// columns wide (32K tokens at stride 16: a tenth of the MMAs, the estimate 147 -> 140 us at the power cap).  Otherwise they
// are neighbouring row tiles of one head.  (128-column tiles, which stream their operands from HBM, do not gain: 205 -> 202
// us for the estimate of 128K tokens, 960 -> 973 us for the prefill.)
//   full[s]   (even CTA)  1 arrival (its producer's expect_tx of both CTAs' bytes) + the bytes of four TMA loads
//   empty[s]  (each CTA)  1 arrival: the commit of the MMAs that read stage s, delivered to both CTAs
//   tfull[a]  (each CTA)  1 arrival: the commit of a tile's last MMA, delivered to both CTAs
//   tempty[a] (even CTA)  8 arrivals: four epilogue warps of each CTA
constexpr int kPairStages = 6;
constexpr int kPairBBytes = 128 * kTileK * 2;                // this CTA's half of the B tile: 16 KiB
constexpr int kPairStageBytes = kABytes + kPairBBytes;       // 32 KiB
constexpr int kPairSmem = kPairStages * kPairStageBytes + 1024 /*barriers*/ + 1024 /*alignment slack*/;

// kDirect: see est_gemm_kernel (0 or 2)
template <int RBS, int kDirect>
__global__ void __launch_bounds__(kGemmThreads, 1)
est_gemm_pair_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmKh,
                     const __grid_constant__ CUtensorMap tmQt, const __grid_constant__ CUtensorMap tmKt,
                     const EstGeom g, const int* group_lo, const int* group_prefix,
                     float* __restrict__ partial, float2* __restrict__ mtile, float* __restrict__ sums, const uint32_t idesc_wide, const uint32_t idesc_narrow,
                     int* status) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ int s_tab[kTabInts];
  if (g.tab_n) {                                  // (made visible by the __syncthreads() that ends the prologue)
    load_tables(g, s_tab);
    group_lo = s_tab + (g.pair_heads ? 0 : kTabPairLo);
    group_prefix = s_tab + (g.pair_heads ? kTabPrefix : kTabPairPrefix);
  }
  // the same offset in both CTAs of the pair (the dynamic shared memory of a kernel starts at the same address
  // in every CTA), which the MMA descriptors rely on
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + kPairStages * kPairStageBytes);
  const uint32_t full0 = smem_u32(bars);                            // [kPairStages]
  const uint32_t empty0 = smem_u32(bars + kPairStages);             // [kPairStages]
  const uint32_t tfull0 = smem_u32(bars + 2 * kPairStages);         // [2]
  const uint32_t tempty0 = smem_u32(bars + 2 * kPairStages + 2);    // [2]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * kPairStages + 4);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);     // (uniform for the compiler too)
  const int lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();                  // 0: issues the MMAs
  const int pair = blockIdx.x >> 1, n_pairs_grid = gridDim.x >> 1;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kPairStages; ++s) {
      mbar_init(full0 + 8 * s, 1);
      mbar_init(empty0 + 8 * s, 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(tfull0 + 8 * a, 1);
      mbar_init(tempty0 + 8 * a, 8);
    }
    *abort_flag = 0;
    fence_mbar_init();
    tma_prefetch_desc(&tmQ);
    tma_prefetch_desc(&tmKh);
  }
  if (warp == 1) {
    tmem_alloc_pair(smem_u32(tmem_slot), 512);
    tmem_relinquish_pair();
  }
  tc_fence_before();
  cluster_sync_all();               // barriers of both CTAs are initialised before any remote arrival or copy
  tc_fence_after();
  pdl_wait();                       // up to here nothing was touched that an earlier kernel writes
  const uint32_t tmem_base = *tmem_slot;

  // row groups of a pair: row tiles of two heads, or pairs of row tiles of one
  const int n_groups = g.pair_heads ? g.n_mtiles : (g.n_mtiles + 1) / 2;
  const int total_tiles = group_prefix[n_groups] * (g.pair_heads ? g.batch * g.hq / 2 : g.batch * g.hq);
  const int k_steps = g.S * g.d_chunks;
  // tile -> this CTA's (batch * head), row tile and column tile; whether the tile is 128 columns wide
  auto decode = [&](int tile, int& bh, int& mt, int& nt) -> bool {
    int grp;
    decode_tile(g, n_groups, group_lo, group_prefix, tile, bh, grp, nt);
    if (!g.pair_heads) {
      mt = 2 * grp + static_cast<int>(rank);
      return false;
    }
    bh = 2 * bh + static_cast<int>(rank);
    mt = grp;
    const int last = mt * kTileM + kTileM - 1 < g.rows_valid - 1 ? mt * kTileM + kTileM - 1 : g.rows_valid - 1;
    int lo, hi;
    row_bounds(g, last, lo, hi);
    return hi - nt * kTileN < 128;
  };

  if (warp == 0) {
    // ------------------------------------------------------------ TMA producer (converged warp, one thread issues)
    {
      const uint32_t lead = elect_one() ? 1u : 0u;
      int s = 0;
      uint32_t ph = 0;
      for (int tile = pair; tile < total_tiles && !*abort_flag; tile += n_pairs_grid) {
        int bh, mt, nt, h, hg_;
        const bool narrow = decode(tile, bh, mt, nt);
        const int b = fast_div(bh, g.by_hq, h), hkv = fast_div(h, g.by_group, hg_);
        const int col0 = nt * g.tile_n + static_cast<int>(rank) * (narrow ? 64 : 128);      // this CTA's columns of B
        const uint32_t stage_bytes = 2 * (kABytes + (narrow ? kPairBBytes / 2 : kPairBBytes));
        int t = 0, dc = 0;
        for (int ks = 0; ks < k_steps; ++ks) {
          if (!__all_sync(0xffffffffu, mbar_wait(empty0 + 8 * s, ph ^ 1, abort_flag))) break;
          const uint32_t dstA = smem_u32(smem + s * kPairStageBytes);
          // all loads of a stage are counted on the even CTA's barrier
          const uint32_t full_even = mapa_shared(full0 + 8 * s, 0);
          mbar_expect_tx_lead(full0 + 8 * s, stage_bytes, rank == 0 ? lead : 0u);
          const bool qt = g.S - 1 - t < g.q_rem, kt = t < g.k_rem;
          const int col = k_column(g, dc);
          load_tile<true>(g, dstA, qt ? &tmQt : &tmQ, full_even, col, g.S - 1 - t, mt * kTileM, h, b, g.q_groups + qt, lead);
          // (B in boxes of 64 columns)
          load_tile<true>(g, dstA + kABytes, kt ? &tmKt : &tmKh, full_even, col, t, col0, hkv, b, g.k_groups + kt, lead);
          load_tile<true>(g, dstA + kABytes + kPairBBytes / 2, kt ? &tmKt : &tmKh, full_even, col, t, col0 + 64, hkv, b, g.k_groups + kt,
                          narrow ? 0u : lead);
          if (++dc == g.d_chunks) { dc = 0; ++t; }
          if (++s == kPairStages) { s = 0; ph ^= 1; }
        }
      }
    }
    // The next kernel comes as the last tiles finish, not before: its CTAs would sit beside this one's for as long as those run, and the
    // block sums are then slower (video diffusion 575 us, 510 like this; presumably as the SM's memory stays divided between cache and
    // shared memory the way this kernel wants it).  us a call, early and like this: 1024 tokens against 70000 101.4 and 97.4, 5000 tokens
    // (estimate and mask, stride 8) 31.25 and 31.10, 32768 tokens (the same, stride 16) 161.0 and 160.4, 20000 tokens 248.5 and 245.1,
    // 60000 tokens at stride 8 1923 and 1911, video diffusion 15361 and 15338; in front of the attention 65536 tokens 494 and 496.
    pdl_launch_dependents();
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer (even CTA; converged warp, one thread issues)
    if (rank == 0) {
      const uint32_t lead = elect_one() ? 1u : 0u;
      auto wait = [&](uint32_t bar, uint32_t ph) { return __all_sync(0xffffffffu, mbar_wait(bar, ph, abort_flag)); };
      int st = 0;
      uint32_t ph = 0, local_tile = 0;
      const uint64_t a_desc0 = smem_desc_sw128(smem_u32(smem), 16, 1024);
      const uint64_t b_desc0 = smem_desc_sw128(smem_u32(smem) + kABytes, 16, 1024);
      for (int tile = pair; tile < total_tiles && !*abort_flag; tile += n_pairs_grid, ++local_tile) {
        int bh_, mt_, nt_;
        const uint32_t idesc = decode(tile, bh_, mt_, nt_) ? idesc_narrow : idesc_wide;
        const uint32_t acc = local_tile & 1;
        const uint32_t acc_ph = (local_tile >> 1) & 1;
        if (!wait(tempty0 + 8 * acc, acc_ph ^ 1)) break;
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + acc * kTileN;
        bool ok = true;
        int term = g.term_chunks ? 0 : -1;
        for (int ks = 0; ks < k_steps; ++ks) {
          if (!wait(full0 + 8 * st, ph)) { ok = false; break; }
          tc_fence_after();
          // D += A of stage sa * B of stage sb; descriptors differ from the stage-0 ones only in the start-address field
          // (units of 16 bytes)
          auto product = [&](int sa, int sb, uint32_t accumulate) {
            const uint64_t a_desc = a_desc0 + static_cast<uint64_t>(sa * (kPairStageBytes >> 4));
            const uint64_t b_desc = b_desc0 + static_cast<uint64_t>(sb * (kPairStageBytes >> 4));
#pragma unroll
            for (int k4 = 0; k4 < kTileK / 16; ++k4)
              mma_ss_pair_lead(d_tmem, a_desc + k4 * 2, b_desc + k4 * 2, idesc, k4 > 0 ? 1u : accumulate, lead);
          };
          if (term < 0) {
            product(st, st, ks > 0 ? 1u : 0u);
            mma_commit_pair_lead(empty0 + 8 * st, 3, lead);       // stage reusable once these MMAs have read it
          } else {
            // three stages hold the terms of one chunk: the products of est_gemm_kernel's fp32 form, each as its terms arrive
            if (term == 0) {
              product(st, st, ks > 0 ? 1u : 0u);
            } else if (term == 1) {
              product(st - 1, st, 1u);
              product(st, st - 1, 1u);
              product(st, st, 1u);
            } else {
              product(st - 2, st, 1u);
              product(st, st - 2, 1u);
              for (int k = 2; k >= 0; --k) mma_commit_pair_lead(empty0 + 8 * (st - k), 3, lead);
            }
            term = term == 2 ? 0 : term + 1;
          }
          if (++st == kPairStages) { st = 0; ph ^= 1; }
        }
        if (!ok) break;
        mma_commit_pair_lead(tfull0 + 8 * acc, 3, lead);  // accumulator complete in both CTAs
      }
    }
  } else {
    // ------------------------------------------------------------ epilogue (4 warps, thread = tile row)
    const int quad = warp & 3;                  // TMEM lane quarter this warp may access
    const int r = quad * 32 + lane;
    const int kGroups = g.tile_n / RBS;         // key blocks per tile
    uint32_t local_tile = 0;
    for (int tile = pair; tile < total_tiles; tile += n_pairs_grid, ++local_tile) {
      int bh, mt, nt;
      const int n_chunks = decode(tile, bh, mt, nt) ? 4 : 8;
      const uint32_t acc = local_tile & 1;
      const uint32_t acc_ph = (local_tile >> 1) & 1;
      const int i = mt * kTileM + r;
      int lo, hi;
      row_bounds(g, i < g.rows_total ? i : g.rows_total, lo, hi);   // rows past the end see nothing
      const int n0 = nt * g.tile_n;
      const int clo = lo - n0 > 0 ? lo - n0 : 0;
      const int chi = hi - n0 < g.tile_n - 1 ? hi - n0 : g.tile_n - 1;
      // warp-uniform: the tensor-memory loads below are warp-collective
      if (!__all_sync(0xffffffffu, mbar_wait(tfull0 + 8 * acc, acc_ph, abort_flag))) break;
      tc_fence_after();
      const uint32_t taddr = tmem_base + acc * kTileN + (static_cast<uint32_t>(quad * 32) << 16);
      // all TMEM reads of this accumulator are done: hand it back to the MMA thread of the even CTA
      auto release = [&]() {
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(mapa_shared(tempty0 + 8 * acc, 0));
      };
      if constexpr (kDirect > 0) {
        const int qb = i / RBS;
        const int out_cols = g.band ? g.bpc : g.kb_total, col0 = g.band ? 0 : nt * kGroups;
        const int nvis = (__reduce_max_sync(0xffffffffu, chi >= clo ? chi : -1) + 32) >> 5;
        int reads = kDirect == 2 && nvis > 4 ? 3 : 1;
        auto load = [&](int half, uint32_t (&v)[4][32]) {
#pragma unroll
          for (int c = 0; c < 4; ++c) tmem_ld32(taddr + half * 128 + c * 32, v[c]);
          tc_wait_ld();
          if (--reads == 0) release();
        };
        est_epilogue_row_direct<RBS, kDirect>(g, load, nvis, clo, chi,
                                        sums + (static_cast<size_t>(bh) * g.qb_total + (qb < g.qb_total ? qb : 0)) * out_cols, col0, out_cols,
                                        qb < g.qb_total, lane);
      } else {
        // (compact scratch: both row tiles of a pair lie in one chunk and start at the pair's first column tile)
        const bool write = mt < g.n_mtiles;
        const size_t tile_at = scratch_tile(g, bh, write ? mt : 0, nt, group_lo[g.pair_heads ? mt : mt / 2]) * kTileM;
        est_epilogue_row<RBS>(g, taddr, n_chunks, clo, chi, write, partial + tile_at * kGroups + r, mtile + tile_at + r, release);
      }
    }
  }

  // ---------------------------------------------------------------- teardown
  tc_fence_before();
  __syncthreads();
  if (*abort_flag) {
    // give copies and MMAs still in flight time to land before shared/tensor memory is released
    const long long t0 = clock64();
    while (clock64() - t0 < 2000000) { __nanosleep(1000); }
    if (threadIdx.x == 0 && status) atomicExch(status, static_cast<int>(kDevWaitTimeout));
  }
  // neither CTA may release tensor memory, or leave while the other can still signal its barriers
  cluster_sync_all();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc_pair(tmem_base, 512);
  }
}

// Normalisation of the partial sums, a CTA per row tile:
//   row i:  m_i = max_t m_{i,t},  l_i = sum_t s_{i,t} 2^(m_{i,t} - m_i)                (m, s = per-tile max and sum)
//   out[kb] = sum_i partial[i][kb] * f_{i,t(kb)},  f_{i,t} = 2^(m_{i,t} - m_i) / l_i
// A stream over the partial sums behind a short chain (statistics, factors): a key block's 128 rows are 512 contiguous bytes that a
// warp reads as one vector per lane, kLines key blocks at a time, the first ones while the statistics are on their way; a lane's four
// rows belong to one query block, whose lanes add by halves.  Bound by HBM where the partial sums do not stay in L2 (video diffusion,
// 119K tokens: 1.33 GB), by latency otherwise.  A warp (or four) per query block read 64 bytes here and there of every key block and
// loaded the next ones only when the ones before were added up.  us between the GEMM's end and the sums', before and now: 119K tokens
// at stride 8 (24 heads) 521 and 284, 32768 at stride 8 17.1 and 12.1, 1024 tokens against 70000 16.7 and 7.9, 9973 9.4 and 5.7.
// kVec > 0: and the selection on the tile's rows of sums, of up to 128 * kVec, from shared memory, a warp per row (select_values; as a
// kernel of its own that is a launch and a hand-over between two kernels more): with the selection 32768 tokens at stride 16
// 18.4 and 14.1, 9973 tokens at stride 8 13.6 and 8.1, 2500 tokens the call 24.8 and 21.0.
// Rows of more than 512 sums go to the selection kernel, whose registers would leave too few warps here.
// Up to two blocks of the selection's values, and the stream, take 64 registers and up to 44 bytes of local memory per thread; without
// those (three quarters of the warps) 5000 tokens 24.6 -> 25.9 us, 8192 at stride 4 36.9 -> 39.0, 32768 at stride 8 244 and 243.
constexpr int kSumGroups = 16;                           // of column tiles: tile t is in group t % 16
constexpr size_t kSumSmem = 84 * 1024;                   // the tile's sums, for the selection: at most 32 rows of 512 and a few more

template <int N>
__device__ __forceinline__ void store_sums(float* p, const float* a) {
  if constexpr (N == 1) *p = a[0];
  else if constexpr (N == 2) *reinterpret_cast<float2*>(p) = make_float2(a[0], a[1]);
  else {
#pragma unroll
    for (int j = 0; j < N; j += 4) *reinterpret_cast<float4*>(p + j) = make_float4(a[j], a[j + 1], a[j + 2], a[j + 3]);
  }
}

template <int RBS, int kVec, int kWarps>
__global__ void __launch_bounds__(32 * kWarps, kVec > 2 ? 24 / kWarps : 32 / kWarps)
est_blocksum_kernel(const EstGeom g, const int* tile_lo, const int* tile_prefix, const float* __restrict__ partial,
                    const float2* __restrict__ mtile, float* __restrict__ sums, int pitch, int split, const EstSelectIf<(kVec > 0)> sel) {
  extern __shared__ __align__(16) float s_rows[];        // (kVec > 0) [query block][pitch], read and written as vectors of four
  __shared__ float4 s_max[kSumGroups][kTileM / 4], s_sum[kSumGroups][kTileM / 4];       // [group][row] of the group's tiles; [0]: of the whole row, and 1 / sum
  constexpr int kLines = RBS == 32 ? 4 : 8;              // key blocks that a warp has in flight (a divisor of a tile's)
  constexpr int kShare = RBS / 4, kLeft = kLines > kShare ? kLines / kShare : 1;      // lanes per query block; sums a lane ends up with
  pdl_launch_dependents();
  pdl_wait();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // the longest row tiles first, in 2^split parts, then those of padding alone
  const int y = blockIdx.y, bh = blockIdx.x, n_real = (g.rows_valid + kTileM - 1) / kTileM;
  const bool pad = y >= n_real << split;
  const int mt = pad ? y - (n_real << split) + n_real : n_real - 1 - (y >> split);
  const int by_parts = pad ? 0 : split, z = y & ((1 << by_parts) - 1);
  const int i0 = mt * kTileM;
  const int nlo = g.tab_n ? g.tab[mt] : tile_lo[mt];
  const int ncnt = g.tab_n ? g.tab[kTabPrefix + mt + 1] - g.tab[kTabPrefix + mt] : tile_prefix[mt + 1] - tile_prefix[mt];
  const int gpt = g.tile_n / RBS, by_gpt = __ffs(gpt) - 1;               // key blocks per tile, a power of two
  const size_t tile0 = scratch_tile(g, bh, mt, nlo, nlo);
  const float4* ms = reinterpret_cast<const float4*>(mtile + tile0 * kTileM) + 2 * lane;        // rows 4 lane .. 4 lane + 3
  const float* pp = partial + tile0 * gpt * kTileM + 4 * lane;                   // key block nlo * gpt + k: at k * kTileM
  const int n_out = g.band ? g.bpc : g.kb_total;
  // key block k is column k + shift(r) of the tile's r-th query block (band layout: only the key blocks of its own chunk are stored)
  auto shift = [&](int r) { return nlo * gpt - (g.band ? (g.row_off + ((i0 + r * RBS) / g.rcs) * g.rcs) / RBS : 0); };
  int k_end = 0;                                         // blocks past the last one that any of the rows sees are zero (and not written by the GEMM)
  if (i0 < g.rows_valid) {
    int lo, hi;
    row_bounds(g, i0 + kTileM - 1 < g.rows_valid - 1 ? i0 + kTileM - 1 : g.rows_valid - 1, lo, hi);
    k_end = hi / RBS + 1 - nlo * gpt;
    if (k_end > ncnt * gpt) k_end = ncnt * gpt;
  }
  float4 p4[kLines];
  float x[4];
  auto fetch = [&](int k0) {                             // the rows of key blocks k0 .. and their (max, sum) in that tile
    const int t = k0 >> by_gpt;
    const float4 a = ld_written(ms + t * (kTileM / 2)), b = ld_written(ms + t * (kTileM / 2) + 1);
    x[0] = a.x; x[1] = a.z; x[2] = b.x; x[3] = b.z;
    const float4* line = reinterpret_cast<const float4*>(pp + static_cast<size_t>(k0) * kTileM);
    if (k0 + kLines <= k_end) {
#pragma unroll
      for (int j = 0; j < kLines; ++j) p4[j] = ld_written_once(line + j * (kTileM / 4));
    } else {
#pragma unroll
      for (int j = 0; j < kLines; ++j) p4[j] = k0 + j < k_end ? ld_written_once(line + j * (kTileM / 4)) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
  };
  // The parts of a row tile: of its key blocks, or (kVec > 0) of the query blocks that are selected on, for which each part adds up all.
  const int k_first = (kVec > 0 ? warp : warp + kWarps * z) * kLines, k_step = (kVec > 0 ? kWarps : kWarps << by_parts) * kLines;
  const int r_first = (warp << by_parts) + z, r_step = kWarps << by_parts;
  if (k_first < k_end) fetch(k_first);
  {
    // The rows' maxima and sums over the tiles, in as many groups whatever the number of warps (the sums do not depend on what else
    // is in the call), then a row per thread over the groups.
#pragma unroll
    for (int i = 0; i < kSumGroups / kWarps; ++i) {
      const int group = warp + i * kWarps;
      float m[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY}, l[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 2
      for (int t = group; t < ncnt; t += kSumGroups) {
        const float4 a = ld_written(ms + t * (kTileM / 2)), b = ld_written(ms + t * (kTileM / 2) + 1);
        const float xm[4] = {a.x, a.z, b.x, b.z}, xl[4] = {a.y, a.w, b.y, b.w};
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          const float mn = fmaxf(m[r], xm[r]);
          // (a tile whose maximum is -inf shows the row nothing, or nothing but NaN, of which its sum would then make the row's)
          if (t == group) l[r] = xm[r] > -INFINITY ? xl[r] : 0.f;
          else if (xm[r] > -INFINITY) l[r] = l[r] * fast_exp2(m[r] - mn) + xl[r] * fast_exp2(xm[r] - mn);
          m[r] = mn;
        }
      }
      s_max[group][lane] = make_float4(m[0], m[1], m[2], m[3]);
      s_sum[group][lane] = make_float4(l[0], l[1], l[2], l[3]);
    }
    __syncthreads();
    if (threadIdx.x < kTileM) {
      float* sm = reinterpret_cast<float*>(s_max) + threadIdx.x;
      float* sl = reinterpret_cast<float*>(s_sum) + threadIdx.x;
      const int groups = ncnt < kSumGroups ? ncnt : kSumGroups;
      float rm = -INFINITY, rl = 0.f;
      for (int w = 0; w < groups; ++w) rm = fmaxf(rm, sm[w * kTileM]);
      if (rm > -INFINITY)
        for (int w = 0; w < groups; ++w) rl += sl[w * kTileM] * fast_exp2(sm[w * kTileM] - rm);
      *sm = rm;
      *sl = rl > 0.f ? 1.f / rl : 0.f;
    }
    __syncthreads();
  }
  const float4 rm4 = s_max[0][lane], ri4 = s_sum[0][lane];
  const float row_m[4] = {rm4.x, rm4.y, rm4.z, rm4.w}, row_inv[4] = {ri4.x, ri4.y, ri4.z, ri4.w};
  const int ql = lane / kShare, part = lane % kShare;    // this lane's query block, and its place among the lanes of it
  const int own_shift = shift(ql);
  float* out = nullptr;
  if constexpr (kVec == 0) out = sums + (static_cast<size_t>(bh) * g.qb_total + i0 / RBS + ql) * n_out;
  const bool real = i0 / RBS + ql < g.qb_total, whole = (reinterpret_cast<uintptr_t>(sums) & 15) == 0;
  const bool aligned = whole && ((n_out | own_shift) & 7) == 0;
#pragma unroll 1
  for (int k0 = k_first; k0 < k_end; k0 += k_step) {
    float f[4], a[kLines];
#pragma unroll
    for (int r = 0; r < 4; ++r) f[r] = row_inv[r] > 0.f ? fast_exp2(x[r] - row_m[r]) * row_inv[r] : 0.f;
#pragma unroll
    for (int j = 0; j < kLines; ++j) a[j] = p4[j].x * f[0] + p4[j].y * f[1] + p4[j].z * f[2] + p4[j].w * f[3];
    if (k0 + k_step < k_end) fetch(k0 + k_step);
    // The sums over a query block's lanes, by halves: a lane gives away half of its sums and receives the other lane's part of
    // the half it keeps.
    int n = kLines, base = 0;
#pragma unroll
    for (int o = kShare / 2; o > 0; o >>= 1) {
      if (n > 1) {
        n >>= 1;
        const bool upper = (part & o) != 0;
        if (upper) base += n;
#pragma unroll
        for (int j = 0; j < kLines / 2; ++j)
          if (j < n) a[j] = (upper ? a[j + n] : a[j]) + __shfl_xor_sync(0xffffffffu, upper ? a[j] : a[j + n], o);
      } else {
        a[0] += __shfl_xor_sync(0xffffffffu, a[0], o);
      }
    }
    const bool writer = kLines >= kShare || (part & (kShare / kLines - 1)) == 0;     // (more lanes than sums)
    const int k = k0 + base;
    if constexpr (kVec > 0) {
      if (writer) store_sums<kLeft>(s_rows + ql * pitch + k, a);
    } else if (writer && real) {
      if (aligned) {
        if (k + own_shift >= 0 && k + own_shift < n_out) store_sums<kLeft>(out + k + own_shift, a);
      } else {
#pragma unroll
        for (int j = 0; j < kLeft; ++j)
          if (k + j + own_shift >= 0 && k + j + own_shift < n_out) out[k + j + own_shift] = a[j];
      }
    }
  }
  const int k_sums = k_end > 0 ? (k_end + kLines - 1) / kLines * kLines : 0;     // of which there are sums; the others are zero
  if constexpr (kVec == 0) {
#pragma unroll 1
    for (int r = r_first; r < kTileM / RBS && i0 / RBS + r < g.qb_total; r += r_step) {
      float* row = sums + (static_cast<size_t>(bh) * g.qb_total + i0 / RBS + r) * n_out;
      const int s = shift(r);
      if (whole && ((n_out | s) & 7) == 0) {
        for (int c = 4 * lane; c < n_out; c += 128)
          if (c - s < 0 || c - s >= k_sums) *reinterpret_cast<float4*>(row + c) = make_float4(0.f, 0.f, 0.f, 0.f);
      } else {
        for (int c = lane; c < n_out; c += 32)
          if (c - s < 0 || c - s >= k_sums) row[c] = 0.f;
      }
    }
  } else {
    __syncthreads();
#pragma unroll 1
    for (int r = r_first; r < kTileM / RBS && i0 / RBS + r < g.qb_total; r += r_step) {
      const int w = bh * g.qb_total + i0 / RBS + r, s = shift(r);
      float* row = sums + static_cast<size_t>(w) * n_out;
      uint32_t v[4 * kVec];
#pragma unroll
      for (int u = 0; u < kVec; ++u) {
        const int c = u * 128 + 4 * lane, k = c - s;
        float e[4] = {0.f, 0.f, 0.f, 0.f};
        if (sel.p.vec_in && (s & 3) == 0) {              // (multiples of four: columns, sums, and where the sums begin)
          if (c < n_out && k >= 0 && k < k_sums) {
            const float4 x4 = *reinterpret_cast<const float4*>(s_rows + r * pitch + k);
            e[0] = x4.x; e[1] = x4.y; e[2] = x4.z; e[3] = x4.w;
          }
        } else {
#pragma unroll
          for (int q = 0; q < 4; ++q)
            if (c + q < n_out && k + q >= 0 && k + q < k_sums) e[q] = s_rows[r * pitch + k + q];
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) v[4 * u + q] = __float_as_uint(e[q]);
        if (sel.p.vec_in) {
          if (c < n_out) *reinterpret_cast<float4*>(row + c) = make_float4(e[0], e[1], e[2], e[3]);
        } else {
#pragma unroll
          for (int q = 0; q < 4; ++q)
            if (c + q < n_out) row[c + q] = e[q];
        }
      }
      select_values<kVec>(v, sel.p, sel.thr_per_head, sel.mask, sel.idx, sel.cnt, w, lane);
    }
  }
}

// fp32 values as rows [hi | mid | lo] of 3 * D bf16 terms, or rounded to bf16 (kTerms == 1).  Rows l >= len_valid are written
// as zeros (a length rounded up to the stride).  Eight elements per thread: two 16-byte loads, a 16-byte store per term.
// HBM-bound: 4 bytes read and 2 or 6 written per element.
template <int kTerms>
__global__ void __launch_bounds__(256)
split_f32_kernel(const float* __restrict__ x, int heads, int len, int len_valid, int vecs, int64_t sb, int64_t sh, int64_t sl,
                 uint4* __restrict__ out, size_t total) {
  pdl_launch_dependents();
  pdl_wait();
  for (size_t e = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; e < total;
       e += static_cast<size_t>(gridDim.x) * blockDim.x) {
    const int d = static_cast<int>(e % vecs);
    size_t rest = e / vecs;
    const int l = static_cast<int>(rest % len);
    rest /= len;
    const int h = static_cast<int>(rest % heads);
    const int b = static_cast<int>(rest / heads);
    unsigned long long v[4] = {};
    if (l < len_valid) {
      const float* row = x + b * sb + h * sh + l * sl + d * 8;
      if ((reinterpret_cast<uintptr_t>(row) & 15) == 0) {
        const float4 a = ld_written_once(reinterpret_cast<const float4*>(row)), c = ld_written_once(reinterpret_cast<const float4*>(row) + 1);
        v[0] = pack_f32x2(a.x, a.y); v[1] = pack_f32x2(a.z, a.w); v[2] = pack_f32x2(c.x, c.y); v[3] = pack_f32x2(c.z, c.w);
      } else {
#pragma unroll
        for (int k = 0; k < 4; ++k) v[k] = pack_f32x2(ld_written(row + 2 * k), ld_written(row + 2 * k + 1));
      }
    }
    uint4* o = out + (e / vecs) * (static_cast<size_t>(kTerms) * vecs) + d;
#pragma unroll
    for (int t = 0; t < kTerms; ++t) o[static_cast<size_t>(t) * vecs] = next_term(v);
  }
}

// The same terms as rows of 6 * D for a product over the widened rows, an element per thread (HBM-bound: 4 bytes read and 12
// written).  role 0: [hi, hi, mid, hi, lo, mid], 1: [hi, mid, hi, lo, hi, mid].
__global__ void __launch_bounds__(256)
split_f32_role_kernel(const float* __restrict__ x, int heads, int len, int len_valid, int D, int64_t sb, int64_t sh, int64_t sl, int role,
                      __nv_bfloat16* __restrict__ out, size_t total) {
  pdl_launch_dependents();
  pdl_wait();
  for (size_t e = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; e < total;
       e += static_cast<size_t>(gridDim.x) * blockDim.x) {
    const int d = static_cast<int>(e % D);
    size_t rest = e / D;
    const int l = static_cast<int>(rest % len);
    rest /= len;
    const int h = static_cast<int>(rest % heads);
    const int b = static_cast<int>(rest / heads);
    const float v = l < len_valid ? ld_written(x + b * sb + h * sh + l * sl + d) : 0.f;
    const __nv_bfloat16 hi = __float2bfloat16_rn(v);
    const float left = v - __bfloat162float(hi);
    const __nv_bfloat16 mid = __float2bfloat16_rn(left), lo = __float2bfloat16_rn(left - __bfloat162float(mid));
    __nv_bfloat16* o = out + (e / D) * (6 * static_cast<size_t>(D)) + d;
    o[0] = hi;
    o[D] = role ? mid : hi;
    o[2 * D] = role ? hi : mid;
    o[3 * D] = role ? lo : hi;
    o[4 * D] = role ? hi : lo;
    o[5 * D] = mid;
  }
}

// ------------------------------------------------------------------------------------ host side
struct EstWorkspace {
  size_t off_tile_lo, off_tile_prefix, off_pair_lo, off_pair_prefix, off_mtile, off_partial;
  size_t total;
};

static int fill_geometry(int batch, int hq, int hkv, int q_len, int k_len, int head_dim, int stride, int block_size,
                         int chunk_size, float scale, int causal, int semantics, EstGeom& g, int step_cols = kTileK) {
  if (batch < 1 || hq < 1 || hkv < 1 || hq % hkv != 0 || q_len < 1 || k_len < 1) return XATTN_B200_ERR_ARG;
  if (stride != 4 && stride != 8 && stride != 16 && stride != 32) return XATTN_B200_ERR_ARG;
  if (block_size != 128 || chunk_size < block_size || chunk_size % block_size != 0) return XATTN_B200_ERR_ARG;
  if (head_dim < step_cols || head_dim % step_cols != 0) return XATTN_B200_ERR_ARG;
  const int k_pad = (chunk_size - k_len % chunk_size) % chunk_size;
  const int q_pad = (chunk_size - q_len % chunk_size) % chunk_size;
  const int lq = q_len + q_pad, lk = k_len + k_pad;
  if (lk / chunk_size < lq / chunk_size) return XATTN_B200_ERR_ARG;   // Xattention.py:39
  g.batch = batch; g.hq = hq; g.hkv = hkv;
  g.by_tiles = make_fast_div(1);
  g.by_group = make_fast_div(hq / hkv);
  g.by_hq = make_fast_div(hq);
  g.S = stride; g.d_chunks = head_dim / step_cols;
  g.rows_total = lq / stride; g.cols_total = lk / stride;
  g.rows_valid = g.rows_total - q_pad / stride;
  g.cols_valid = g.cols_total - k_pad / stride;
  g.rcs = chunk_size / stride;
  g.row_off = (lk / chunk_size - lq / chunk_size) * g.rcs;
  g.causal = causal ? 1 : 0;
  g.left_blank = (causal && semantics != XATTN_B200_SEMANTICS_TRITON && k_pad / stride == 0) ? 1 : 0;
  g.band = semantics == XATTN_B200_SEMANTICS_TORCH_BAND ? 1 : 0;
  g.bpc = chunk_size / block_size;
  if (g.band && !g.left_blank) return XATTN_B200_ERR_ARG;
  g.rbs = block_size / stride;
  g.kb_total = lk / block_size; g.qb_total = lq / block_size;
  g.n_mtiles = (g.rows_total + kTileM - 1) / kTileM;
  // narrow tiles when every row sees at most one 128-column span (torch branch with chunk_size <= 128*stride):
  // a 256-wide tile would spend half of its MMA work on hidden columns
  // (and when the keys have no more than 128 columns at all)
  g.tile_n = ((g.left_blank && g.rcs <= 128) || (g.causal ? g.cols_valid : g.cols_total) <= 128) ? 128 : kTileN;
  g.n_ntiles = (g.cols_total + g.tile_n - 1) / g.tile_n;
  g.scale_log2 = scale * 1.4426950408889634f;
  g.head_dim = head_dim;
  g.tab_n = 0;
  g.term_chunks = 0;
  g.q_rem = q_len % stride;
  g.k_rem = k_len % stride;
  g.q_groups = q_len / stride;
  g.k_groups = k_len / stride;
  g.row_cols = head_dim;
  g.direct = 0;
  g.split = 1;
  g.pair_heads = 0;
  g.compact = g.left_blank;
  g.m_pitch = g.n_ntiles;
  if (g.compact) {
    int max_cnt = 1;
    for (int mt = 0; mt < g.n_mtiles; ++mt) {
      int first, cnt;
      row_tile_range(g, mt, first, cnt);
      max_cnt = cnt > max_cnt ? cnt : max_cnt;
    }
    g.m_pitch = max_cnt;
  }
  return XATTN_B200_OK;
}

static EstWorkspace workspace_layout(const EstGeom& g) {
  EstWorkspace w;
  auto up = [](size_t x) { return (x + 255) & ~size_t(255); };
  size_t o = 0;
  w.off_tile_lo = o; o = up(o + sizeof(int) * g.n_mtiles);
  w.off_tile_prefix = o; o = up(o + sizeof(int) * (g.n_mtiles + 1));
  w.off_pair_lo = o; o = up(o + sizeof(int) * ((g.n_mtiles + 1) / 2));
  w.off_pair_prefix = o; o = up(o + sizeof(int) * ((g.n_mtiles + 1) / 2 + 1));
  const size_t rows = static_cast<size_t>(g.batch) * g.hq * g.n_mtiles * kTileM;
  w.off_mtile = o; o = up(o + sizeof(float2) * rows * g.m_pitch);
  w.off_partial = o; o = up(o + sizeof(float) * rows * g.m_pitch * (g.tile_n / g.rbs));
  w.total = o;
  return w;
}

// Scratch of one estimate call: exact for the given mask and semantics, or (causal < 0) enough for any.
size_t estimate_workspace_bytes(int batch, int hq, int q_len, int k_len, int stride, int block_size, int chunk_size,
                                int causal, int semantics) {
  auto bytes = [&](int c, int sem) -> size_t {           // (neither head_dim nor hkv changes the layout)
    EstGeom g;
    const int rc = fill_geometry(batch, hq, hq, q_len, k_len, 128, stride, block_size, chunk_size, 1.f, c, sem, g);
    return rc == XATTN_B200_OK ? workspace_layout(g).total : 0;
  };
  if (causal >= 0) return bytes(causal, semantics);
  // The causal torch layout is the compact one, and not always the smaller: chunks of one and a half 128-column tiles make row
  // tiles span two of them where the other layouts have a single 256-column tile.
  const size_t need[] = {bytes(0, XATTN_B200_SEMANTICS_TORCH), bytes(1, XATTN_B200_SEMANTICS_TRITON), bytes(1, XATTN_B200_SEMANTICS_TORCH)};
  const size_t most = need[0] > need[1] ? need[0] : need[1];
  return most > need[2] ? most : need[2];
}

// Of that, what the rows of the call take without their padding to whole tiles (0: refused arguments).
size_t estimate_row_bytes(int batch, int hq, int q_len, int k_len, int stride, int block_size, int chunk_size, int causal, int semantics) {
  EstGeom g;
  if (fill_geometry(batch, hq, hq, q_len, k_len, 128, stride, block_size, chunk_size, 1.f, causal, semantics, g) != XATTN_B200_OK) return 0;
  const size_t pairs = g.compact ? g.m_pitch : (g.cols_total + kTileN - 1) / kTileN;
  const size_t sums = g.compact ? pairs * (g.tile_n / g.rbs) : g.kb_total;
  return static_cast<size_t>(batch) * hq * g.rows_total * (sizeof(float2) * pairs + sizeof(float) * sums);
}

int split_f32_launch(const float* x, int batch, int heads, int len, int len_valid, int head_dim, int64_t sb, int64_t sh,
                     int64_t sl, int terms, void* out, cudaStream_t stream);

// CTA pairs (256x256 tiles) when tiles are 256 columns wide and the two row tiles of a pair see about the
// same columns (always, except when a 128-row chunk of the torch branch blanks everything left of it)
static bool pairs_fit(const EstGeom& g) { return g.tile_n == kTileN && g.n_mtiles >= 2 && (!g.left_blank || g.rcs % (2 * kTileM) == 0); }

// Whether the estimate of fp32 inputs is better done from rows of bf16 terms, written once, than by splitting the values as each
// tile is loaded.  The terms cost a pass over HBM of 10 bytes per element, and the GEMM of a tile then takes half the time (CTA
// pairs; the split is bound by shared memory and the latency of its steps): with T tiles of 128 x 256 per head that half is about
// T * stride * 0.026 us, the pass 0.00023 us per token and head.  Measured (32 heads; estimate alone; terms, split in the GEMM):
// 4096 tokens at stride 16 134, 81 us; 8192 at 16 288, 243; 8192 at 8 334, 317, with 8 kv heads 274, 317.
int estimate_f32_terms(int hq, int hkv, int q_len, int k_len, int stride, int block_size, int chunk_size, int causal, int semantics) {
  EstGeom g;
  if (fill_geometry(1, hq, hkv, q_len, k_len, 128, stride, block_size, chunk_size, 1.f, causal, semantics, g) || !pairs_fit(g)) return 0;
  long long tiles = 0;
  for (int mt = 0; mt < g.n_mtiles; ++mt) {
    int first, count;
    row_tile_range(g, mt, first, count);
    tiles += count;
  }
  return tiles * stride * 105 > q_len + static_cast<long long>(k_len) * hkv / hq;
}

int estimate_launch(const void* q, const void* k, int dtype, int batch, int hq, int hkv, int q_len, int k_len,
                    int head_dim, int64_t qsb, int64_t qsh, int64_t qsl, int64_t ksb, int64_t ksh, int64_t ksl,
                    int stride, int block_size, int chunk_size, float scale, int causal, int semantics,
                    float* attn_sums, void* workspace, size_t workspace_bytes, void* q_bf16, void* k_bf16, int* status,
                    cudaStream_t stream, const SelCall* select, bool* selected) {
  const bool f32 = dtype == XATTN_B200_F32, terms = dtype == XATTN_B200_F32_TERMS;
  if (!q || !k || !attn_sums) return XATTN_B200_ERR_ARG;
  if (dtype != XATTN_B200_BF16 && dtype != XATTN_B200_F16 && !f32 && !terms) return XATTN_B200_ERR_ARG;
  if ((q_bf16 || k_bf16) && (!f32 || !q_bf16 || !k_bf16 || ((reinterpret_cast<uintptr_t>(q_bf16) | reinterpret_cast<uintptr_t>(k_bf16)) & 15)))
    return XATTN_B200_ERR_ARG;
  if (semantics != XATTN_B200_SEMANTICS_TORCH && semantics != XATTN_B200_SEMANTICS_TRITON &&
      semantics != XATTN_B200_SEMANTICS_TORCH_BAND)
    return XATTN_B200_ERR_ARG;
  if (!(scale > 0.f)) return XATTN_B200_ERR_ARG;
  EstGeom g;
  int rc = fill_geometry(batch, hq, hkv, q_len, k_len, head_dim, stride, block_size, chunk_size, scale, causal,
                         semantics, g, f32 ? kF32Cols : kTileK);
  if (rc) return rc;
  if (terms) {
    // (the terms are written for whole stride groups; geometries without CTA pairs take fp32 rows)
    if (q_len % stride || k_len % stride || !pairs_fit(g)) return XATTN_B200_ERR_ARG;
    g.row_cols = 3 * head_dim;
    g.term_chunks = g.d_chunks;
    g.d_chunks *= 3;
  }
  const EstWorkspace w = workspace_layout(g);
  if (!workspace || workspace_bytes < w.total) return XATTN_B200_ERR_WORKSPACE;
  if ((rc = check_sm100())) return rc;
  // every stated maximum is checked before the first launch, so that a refusal leaves no work in flight
  const long long total_rows = static_cast<long long>(batch) * hq * g.rows_total;
  if (g.n_mtiles > 8192 || total_rows > 0x7fffffffLL || static_cast<long long>(batch) * hq > 65535 ||
      g.qb_total > 65535)
    return XATTN_B200_ERR_LIMIT;

  uint8_t* ws = static_cast<uint8_t*>(workspace);
  int* tile_lo = reinterpret_cast<int*>(ws + w.off_tile_lo);
  int* tile_prefix = reinterpret_cast<int*>(ws + w.off_tile_prefix);
  int* pair_lo = reinterpret_cast<int*>(ws + w.off_pair_lo);
  int* pair_prefix = reinterpret_cast<int*>(ws + w.off_pair_prefix);
  float2* mtile = reinterpret_cast<float2*>(ws + w.off_mtile);
  float* partial = reinterpret_cast<float*>(ws + w.off_partial);

  // 5-D views [head_dim, S, len/S, heads, batch] whose second coordinate picks the token inside a stride group; `tail`: with
  // the ragged last group and the token offsets it has (see EstGeom::q_rem).  No map describes a token that does not exist.
  auto make_map = [&](CUtensorMap* m, const void* x, int len, int heads, int64_t sb, int64_t sh, int64_t sl, uint32_t box_rows, bool tail) -> int {
    if (len < stride) tail = true;                       // (no whole group: the map is never loaded from in its bounds)
    const int offsets = tail ? len % stride : stride, groups = len / stride + (tail ? 1 : 0);
    const uint64_t dims[5] = {(uint64_t)g.row_cols, (uint64_t)offsets, (uint64_t)groups, (uint64_t)heads, (uint64_t)batch};
    // a dimension of extent 1 never moves: give it a harmless valid stride
    const uint64_t e = f32 ? 4 : 2;
    const uint64_t str[4] = {(uint64_t)sl * e, (uint64_t)sl * e * stride, heads > 1 ? (uint64_t)sh * e : 256, batch > 1 ? (uint64_t)sb * e : 256};
    const uint32_t box[5] = {static_cast<uint32_t>(f32 ? kF32Cols : kTileK), 1, box_rows, 1, 1};
    return make_tmap(m, x, f32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 5, dims, str, box);
  };

  bool use_pairs = pairs_fit(g);
  g.pair_heads = g.tile_n == kTileN && (hq / hkv) % 2 == 0 ? 1 : 0;
  if (g.pair_heads) use_pairs = true;
  if (f32) use_pairs = false;
  bool many = false;                                       // more than four tiles per SM
  // Few tiles (short prompts: 32 heads of up to 2048 tokens at stride 16 are 32 tiles for 148 SMs): the K loop of each, which is
  // a stream of operands through one SM, is split over a cluster of two or four CTAs instead.
  {
    long long tiles = 0;
    for (int mt = 0; mt < g.n_mtiles && tiles <= 4LL * sm_count(); ++mt) {
      int first, count;
      row_tile_range(g, mt, first, count);
      tiles += static_cast<long long>(count > 0 ? count : 1) * batch * hq;
    }
    many = tiles > 4LL * sm_count();
    const bool long_k = g.S * g.d_chunks >= 32 && !terms;          // (the exchange costs about what eight steps take)
    g.split = !long_k ? 1 : (4 * tiles <= sm_count() ? 4 : (2 * tiles <= sm_count() ? 2 : 1));
    if (g.split > 1) use_pairs = false;
    if (!use_pairs) g.pair_heads = 0;
  }
  // Every row sees a single column tile, and that tile's block sums are (nearly) a whole row of the output: chunks of exactly
  // 128 or 256 reshaped rows in the chunk-band layout (128K or 64K tokens at stride 16), or keys of at most 256 columns
  // altogether (prompts of up to 4096 tokens at stride 16) or of a few such chunks.  The GEMM's epilogue then finishes the block sums itself, and
  // neither the scratch arrays nor est_blocksum_kernel are needed.
  bool direct = g.rbs <= 32 && 32 % g.rbs == 0;
  if (g.band)
    direct = direct && g.compact && g.m_pitch == 1 && g.rcs == g.tile_n && g.row_off % g.tile_n == 0 && g.bpc == g.tile_n / g.rbs;
  else
    direct = direct && g.kb_total <= 8 * g.tile_n / g.rbs;             // (the epilogue writes the zeros, a few at a time)
  for (int mt = 0; direct && mt < g.n_mtiles; ++mt) {
    int first, count;
    row_tile_range(g, mt, first, count);
    direct = g.band ? count == 1 && first * g.tile_n == (mt * kTileM / g.rcs) * g.rcs + g.row_off : count <= 1;
  }
  g.direct = direct ? 1 : 0;
  // Block sums finished there can be selected on there, too: rows of up to 128 stored sums (four per lane), in clusters of four, or
  // where a CTA has tiles enough that the selection on one runs under the next.  Clusters of two do not gain: a CTA has the rows of
  // eight query blocks at stride 16, two rounds for its six warps (2100 tokens 35.4 us a call with it, 35.2 without).  Otherwise
  // est_blocksum_kernel selects, rows of up to 512 whose tile fits its shared memory.
  EstSelect sel;
  bool selecting = false;
  if (select) {
    const SelCall& c = *select;
    const int cols = g.band ? g.bpc : g.kb_total;
    const bool here = direct ? !use_pairs && can_select(g.tile_n / 128, f32) && (g.split == 4 || (g.split == 1 && many)) && cols <= 128
                             : cols <= 512 && static_cast<size_t>(kTileM / g.rbs) * (g.m_pitch * (g.tile_n / g.rbs) + 8) * sizeof(float) <= kSumSmem;
    if (here && c.k_blocks <= 1024 && c.attn_sums == attn_sums && c.batch == batch && c.heads == hq && c.q_blocks == g.qb_total &&
        c.k_blocks == g.kb_total && c.bpc == g.bpc && (c.band ? 1 : 0) == g.band) {
      if ((rc = select_params(c, sel.p))) return rc;
      selecting = true;
      sel.thr_per_head = c.thr_per_head;
      sel.mask = c.mask;
      sel.idx = c.block_idx;
      sel.cnt = c.block_cnt;
      *selected = true;
    }
  }
  CUtensorMap tmQ, tmK, tmQt, tmKt;
  const uint32_t k_box = use_pairs ? 64 : (f32 ? static_cast<uint32_t>(kTileM) : static_cast<uint32_t>(g.tile_n));
  if ((rc = make_map(&tmQ, q, q_len, hq, qsb, qsh, qsl, kTileM, false))) return rc;
  if ((rc = make_map(&tmK, k, k_len, hkv, ksb, ksh, ksl, k_box, false))) return rc;
  tmQt = tmQ;
  tmKt = tmK;
  if (g.q_rem && (rc = make_map(&tmQt, q, q_len, hq, qsb, qsh, qsl, kTileM, true))) return rc;
  if (g.k_rem && (rc = make_map(&tmKt, k, k_len, hkv, ksb, ksh, ksl, k_box, true))) return rc;

  // The tile tables (the arithmetic of est_setup_kernel): their totals, and, for few row tiles, the tables themselves, which
  // then travel in the kernel parameters.
  const bool in_params = g.n_mtiles <= kTabTiles;
  // up to 64 KiB of dynamic shared memory (8192 row tiles): above the 48 KiB a kernel gets without asking
  if (!in_params && !allow_smem(est_setup_kernel, 2 * sizeof(int) * 8192)) return XATTN_B200_ERR_CUDA;
  int tiles_per_head = 0, pairs_per_head = 0;
  for (int mt = 0, lo = 0, hi = -1; mt < g.n_mtiles; ++mt) {
    int first, cnt;
    row_tile_range(g, mt, first, cnt);
    if (mt % 2 == 0) {
      lo = 0x7fffffff;
      hi = -1;
    }
    if (cnt > 0 && counts_in_pair(g, mt)) {
      lo = first < lo ? first : lo;
      hi = first + cnt - 1 > hi ? first + cnt - 1 : hi;
    }
    if (in_params) {
      g.tab[mt] = first;
      g.tab[kTabPrefix + mt] = tiles_per_head;
      g.tab[kTabPairLo + mt / 2] = hi < 0 ? 0 : lo;
      g.tab[kTabPairPrefix + mt / 2] = pairs_per_head;
    }
    tiles_per_head += cnt;
    if (mt % 2 == 1 || mt == g.n_mtiles - 1) pairs_per_head += hi < 0 ? 0 : hi - lo + 1;
  }
  const int per_head = use_pairs && !g.pair_heads ? pairs_per_head : tiles_per_head;
  g.by_tiles = make_fast_div(static_cast<uint32_t>(per_head > 0 ? per_head : 1));
  if (static_cast<long long>(tiles_per_head) * batch * hq > 0x7fffffffLL) return XATTN_B200_ERR_LIMIT;
  if (in_params) {
    g.tab[kTabPrefix + g.n_mtiles] = tiles_per_head;
    g.tab[kTabPairPrefix + (g.n_mtiles + 1) / 2] = pairs_per_head;
    g.tab_n = g.n_mtiles;
  } else if ((rc = launch_dependent(est_setup_kernel, dim3(1), dim3(256), 2 * sizeof(int) * g.n_mtiles, stream, g, tile_lo, tile_prefix,
                                    pair_lo, pair_prefix))) {
    return rc;
  }

  const int sms = sm_count();
  if (use_pairs) {
    const uint32_t idesc2 = make_idesc_f16(2 * kTileM, kTileN, dtype != XATTN_B200_F16, false, false);
    const uint32_t idesc2n = make_idesc_f16(2 * kTileM, 128, dtype != XATTN_B200_F16, false, false);
    auto launch_pair = [&](auto kern) -> int {
      if (!allow_smem(kern, kPairSmem))
        return XATTN_B200_ERR_CUDA;
      cudaLaunchConfig_t cfg = {};
      cfg.gridDim = dim3(static_cast<unsigned>(sms & ~1), 1, 1);
      cfg.blockDim = dim3(kGemmThreads, 1, 1);
      cfg.dynamicSmemBytes = kPairSmem;
      cfg.stream = stream;
      cudaLaunchAttribute attr[1];
      attr[0].id = cudaLaunchAttributeClusterDimension;
      attr[0].val.clusterDim.x = 2;
      attr[0].val.clusterDim.y = 1;
      attr[0].val.clusterDim.z = 1;
      cfg.attrs = attr;
      cfg.numAttrs = 1;
      // every pair must be resident at once (persistent kernel): shrink the grid to what the device can hold
      const int max_clusters = once_per_device(reinterpret_cast<const void*>(kern), [&]() {
        int m = 0;
        return cudaOccupancyMaxActiveClusters(&m, kern, &cfg) == cudaSuccess ? m : 0;
      });
      if (max_clusters < 1) return XATTN_B200_ERR_CUDA;
      if (static_cast<unsigned>(2 * max_clusters) < cfg.gridDim.x) cfg.gridDim.x = 2 * max_clusters;
      return launch_dependent_clusters(kern, 2, cfg.gridDim, cfg.blockDim, kPairSmem, stream, tmQ, tmK, tmQt, tmKt, g,
                                       (const int*)(g.pair_heads ? tile_lo : pair_lo), (const int*)(g.pair_heads ? tile_prefix : pair_prefix),
                                       partial, mtile, attn_sums, idesc2, idesc2n, status);
    };
    auto launch_pair_rbs = [&](auto rbs) -> int {
      constexpr int kRbs = decltype(rbs)::value;
      if (!direct) return launch_pair(est_gemm_pair_kernel<kRbs, 0>);
      return launch_pair(est_gemm_pair_kernel<kRbs, 2>);
    };
    switch (g.rbs) {
      case 4: rc = launch_pair_rbs(std::integral_constant<int, 4>()); break;
      case 8: rc = launch_pair_rbs(std::integral_constant<int, 8>()); break;
      case 16: rc = launch_pair_rbs(std::integral_constant<int, 16>()); break;
      case 32: rc = launch_pair_rbs(std::integral_constant<int, 32>()); break;
      default: rc = XATTN_B200_ERR_ARG;
    }
    if (rc || direct) return rc;                       // (direct: the block sums are complete)
  } else {
  const uint32_t idesc = make_idesc_f16(kTileM, g.tile_n, dtype != XATTN_B200_F16, false, false);
  // persistent CTAs, or exactly the tiles' clusters
  const long long tiles = static_cast<long long>(tiles_per_head) * batch * hq;
  if (tiles == 0) g.split = 1;
  const int grid = g.split > 1 ? static_cast<int>(tiles) * g.split : sms;
  // The roundings of fp32 operands come with the tiles: a row tile's with its first, a column tile's with the first row tile that
  // has it.  Where that leaves tokens out (keys that no query of the call may see), they are written by a pass of their own.
  EstRounded rounded = {static_cast<uint4*>(q_bf16), static_cast<uint4*>(k_bf16), q_len, k_len};
  if (q_bf16) {
    int q_tokens = 0, k_tokens = 0, last = 0;            // the tokens before these are covered
    for (int mt = 0; mt < g.n_mtiles; ++mt) {
      int first, cnt;
      row_tile_range(g, mt, first, cnt);
      if (cnt > 0 && q_tokens == mt * kTileM * g.S) q_tokens += kTileM * g.S;
      if (cnt > 0 && first <= last) last = first + cnt > last ? first + cnt : last;
    }
    k_tokens = last * g.tile_n * g.S;
    if (q_tokens < q_len) {
      if ((rc = split_f32_launch(static_cast<const float*>(q), batch, hq, q_len, q_len, head_dim, qsb, qsh, qsl, 1, q_bf16, stream))) return rc;
      rounded.q = nullptr;
    }
    if (k_tokens < k_len) {
      if ((rc = split_f32_launch(static_cast<const float*>(k), batch, hkv, k_len, k_len, head_dim, ksb, ksh, ksl, 1, k_bf16, stream))) return rc;
      rounded.k = nullptr;
    }
  }
  auto launch = [&](auto kern, int threads, int smem, auto what) -> int {
    if (!allow_smem(kern, smem)) return XATTN_B200_ERR_CUDA;
    return launch_dependent_clusters(kern, g.split, dim3(grid), dim3(threads), smem, stream, tmQ, tmK, tmQt, tmKt, g, (const int*)tile_lo,
                                     (const int*)tile_prefix, partial, mtile, attn_sums, idesc, rounded, what, status);
  };
  auto launch_type = [&](auto rbs, auto halves) -> int {
    constexpr int kRbs = decltype(rbs)::value, kDirect = decltype(halves)::value;
    if constexpr (can_select(kDirect, false)) {
      if (selecting) return launch(est_gemm_kernel<kRbs, kDirect, false, true>, kGemmThreads, kGemmSmem, sel);
    }
    return f32 ? launch(est_gemm_kernel<kRbs, kDirect, true, false>, f32_threads(kDirect), kF32Smem + 2048, EstNothing())
               : launch(est_gemm_kernel<kRbs, kDirect, false, false>, kGemmThreads, kGemmSmem, EstNothing());
  };
  auto launch_rbs = [&](auto rbs) -> int {
    if (!direct) return launch_type(rbs, std::integral_constant<int, 0>());
    return g.tile_n == 128 ? launch_type(rbs, std::integral_constant<int, 1>()) : launch_type(rbs, std::integral_constant<int, 2>());
  };
  switch (g.rbs) {
    case 4: rc = launch_rbs(std::integral_constant<int, 4>()); break;
    case 8: rc = launch_rbs(std::integral_constant<int, 8>()); break;
    case 16: rc = launch_rbs(std::integral_constant<int, 16>()); break;
    case 32: rc = launch_rbs(std::integral_constant<int, 32>()); break;
    default: rc = XATTN_B200_ERR_ARG;
  }
  if (direct) return rc;                               // the block sums are complete
  if (rc) return rc;
  }

  const int gpt = g.tile_n / g.rbs, pitch = g.m_pitch * gpt + 8;        // (rows of sums in different banks)
  // Few row tiles (of those that hold rows: a short piece of prompt is padded to a chunk) are divided over CTAs.  Where they are selected
  // on, each part adds up all of the sums, which is little, and selects on some of the query blocks: a long selection by sixteen warps of
  // one SM is slow.  As long as a part has more than four (rows of up to 128 sums: eight, which are done soon, and the attention
  // kernel sets up on the SMs left: 2048 tokens of 28 heads at stride 8 35.7 us with four, 35.1), and up to a CTA per SM, or two where there
  // would be two rounds of warps.  Otherwise a part has some of the key blocks, up to two CTAs per SM.  us a call, 32 heads, flat scores, one CTA
  // per row tile and like this: 2048 tokens against 30000 at stride 32 53.9 and 43.4, at stride 8 53.6 and 41.2, 12000 at stride 32 58.4 and 49.0, 2048
  // against 131072 56.7 and 54.6; 1024 against 70000 100 and 82 (padding counted and not).
  const int real_tiles = (g.rows_valid + kTileM - 1) / kTileM;
  const unsigned sum_ctas = static_cast<unsigned>(batch) * hq * real_tiles;
  const int tile_rows = ((g.rows_valid < kTileM ? g.rows_valid : kTileM) + g.rbs - 1) / g.rbs;      // query blocks of a row tile
  const int cols = g.band ? g.bpc : g.kb_total;
  int split = 0;
  if (selecting)
    while (tile_rows > (cols > 128 ? 4 : 8) << split && sum_ctas << (split + 1) <= (tile_rows > 16 << split ? 2u : 1u) * sms) ++split;
  else
    while (split < 3 && sum_ctas << (split + 1) <= 2u * sms) ++split;
  // Sixteen warps where that leaves no more than two CTAs per SM, otherwise eight; eight, too, for a few sums in front of the selection
  // kernel, whose CTAs then find registers free and set up under them (1024 tokens against 131072, 16 key blocks visible: 29.6 and 26.4;
  // 512 against 300000, 2344 key blocks: 244 and 259).
  const bool wide = sum_ctas <= 2u * sms && !(select && !selecting && pitch >> split <= 64);
  auto launch_sums = [&](auto kern, int threads, auto what) -> int {
    const size_t smem = selecting ? static_cast<size_t>(kTileM / g.rbs) * pitch * sizeof(float) : 0;
    if (smem > 24 * 1024 && !allow_smem(kern, kSumSmem)) return XATTN_B200_ERR_CUDA;
    return launch_dependent(kern, dim3(static_cast<unsigned>(batch) * hq, (real_tiles << split) + g.n_mtiles - real_tiles), dim3(threads), smem, stream, g, (const int*)tile_lo,
                            (const int*)tile_prefix, (const float*)partial, (const float2*)mtile, attn_sums, pitch, split, what);
  };
  // with the selection: the instantiation with just enough registers for a row of sums
  auto launch_vec = [&](auto rbs, auto warps) -> int {
    constexpr int kRbs = decltype(rbs)::value, kWarps = decltype(warps)::value;
    if (!selecting) return launch_sums(est_blocksum_kernel<kRbs, 0, kWarps>, 32 * kWarps, EstNothing());
    if (cols <= 128) return launch_sums(est_blocksum_kernel<kRbs, 1, kWarps>, 32 * kWarps, sel);
    if (cols <= 256) return launch_sums(est_blocksum_kernel<kRbs, 2, kWarps>, 32 * kWarps, sel);
    return launch_sums(est_blocksum_kernel<kRbs, 4, kWarps>, 32 * kWarps, sel);
  };
  auto launch_team = [&](auto rbs) -> int {
    return wide ? launch_vec(rbs, std::integral_constant<int, 16>()) : launch_vec(rbs, std::integral_constant<int, 8>());
  };
  switch (g.rbs) {
    case 4: return launch_team(std::integral_constant<int, 4>());
    case 8: return launch_team(std::integral_constant<int, 8>());
    case 16: return launch_team(std::integral_constant<int, 16>());
    case 32: return launch_team(std::integral_constant<int, 32>());
    default: return XATTN_B200_ERR_ARG;
  }
}

int split_f32_launch(const float* x, int batch, int heads, int len, int len_valid, int head_dim, int64_t sb, int64_t sh,
                     int64_t sl, int terms, void* out, cudaStream_t stream) {
  if (!x || !out || batch < 1 || heads < 1 || len < 1 || len_valid < 1 || len_valid > len || head_dim < 8 || head_dim % 8 ||
      (terms != 1 && terms != 3) || (reinterpret_cast<uintptr_t>(out) & 15))
    return XATTN_B200_ERR_ARG;
  const size_t total = static_cast<size_t>(batch) * heads * len * (head_dim / 8);
  const int block = 256;
  const size_t most = 32 * static_cast<size_t>(sm_count());
  size_t blocks = (total + block - 1) / block;
  if (blocks > most) blocks = most;
  auto launch = [&](auto kern) -> int {
    return launch_dependent(kern, dim3(static_cast<unsigned>(blocks)), dim3(block), 0, stream, x, heads, len, len_valid, head_dim / 8, sb,
                            sh, sl, static_cast<uint4*>(out), total);
  };
  return terms == 3 ? launch(split_f32_kernel<3>) : launch(split_f32_kernel<1>);
}

int split_f32_role_launch(const float* x, int batch, int heads, int len, int len_valid, int head_dim, int64_t sb, int64_t sh,
                          int64_t sl, int role, void* out, cudaStream_t stream) {
  if (!x || !out || batch < 1 || heads < 1 || len < 1 || len_valid < 1 || len_valid > len || head_dim < 1 || (role != 0 && role != 1))
    return XATTN_B200_ERR_ARG;
  const size_t total = static_cast<size_t>(batch) * heads * len * head_dim, cap = 32 * static_cast<size_t>(sm_count());
  const size_t blocks = (total + 255) / 256;
  return launch_dependent(split_f32_role_kernel, dim3(static_cast<unsigned>(blocks < cap ? blocks : cap)), dim3(256), 0, stream, x, heads, len,
                          len_valid, head_dim, sb, sh, sl, role, static_cast<__nv_bfloat16*>(out), total);
}

}  // namespace xb
