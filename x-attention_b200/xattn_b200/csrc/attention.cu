// Phase 3 of the XAttention prefill path: block-sparse FlashAttention forward over 128x128 blocks.
//
// Replaces block_sparse_attn.block_sparse_attn_func (third-party CUDA package; call site
// xattn/src/Xattention.py:377-391).  A tile is one (batch, head, 128-row query block) with its list of kept key
// blocks (or, for dense calls, the blocks 0 .. n-1 without a list in memory).  A unit of work is two tiles that read the
// same kv head: two query heads of a kv group, or two neighbouring query blocks of one head.  The grid has a CTA per
// unit, of which one per SM runs at a time and takes over further ones (cluster launch control).  Its two tiles are two
// streams: each has its own Q tile in shared memory, its own score/probability buffer S and output accumulator O in
// tensor memory and its own softmax warpgroup, so that one stream's softmax runs under the other's MMAs.  (Calls of few tiles: a
// unit is a single tile, of whose list each stream walks every other block, and the epilogue adds the two parts of O.  Only the pass over
// what the pair kernel leaves, whose length the host does not know, takes its units in strides of the grid instead.)
//
//   warps 0-3   softmax of stream 0  } one thread per query row.  A block's 128 scores leave TMEM once and stay in
//   warps 4-7   softmax of stream 1  } registers for the row maximum (3-input max) and the exp2; P packed to 16-bit
//                                      goes back into S columns, handed to the tensor pipe in two halves; lazy
//                                      rescale of O only when the max grew by more than 2^8; the row sum of the
//                                      tile's last block goes to shared memory for the epilogue
//   warps 8-11  epilogue of both streams: O / l from TMEM, through shared memory, to TMA stores
//   warp  12    loader of K and V: the union of the two lists passes once through a ring of two K and two V slots that
//               both streams read; requests the units of work
//   warp  13    tcgen05 issuer of both streams: S = Q K^T (operands in shared memory), then O += P V (P from TMEM, V
//               from shared memory as an MN-major operand)
//   warp  14    loader of Q
//
// What bounds it, and what follows from that (dense causal mask, 32 heads x 16384 tokens: 1110 -> 1372 TFLOP/s; 32768
// tokens with 2.5 listed blocks per row: 254 -> 166 us in short runs):
//   * A 128x128 block is 1024 cycles of MMA and 1024 cycles of ex2 (16 per cycle and SM), so the two streams have to be
//     half a period apart.  One warp issues the MMAs of both in fixed alternation: a stream's batch then goes through
//     the tensor pipe in one piece.  Two issuing warps' batches interleave, both streams' scores are complete at the
//     same time, both exponentiate at half speed, and the tensor pipe idles.
//   * tcgen05 takes its operands from uniform registers.  Issued from a single-thread branch an MMA cost 83 cycles, more
//     than its 64 cycles of work; issued under a predicate in converged code, 10.
//   * Shared memory (128 B per cycle) has to take the operand reads of Q.K^T (64 KiB a block), of P.V (32 KiB) and the TMA
//     writes of K and V (64 KiB if every tile brings its own): 1280 cycles, against 1024 when two tiles share them; and
//     L2 delivers half the bytes.
//   * Short lists walk through all of the code every few microseconds.  At 74 KB of code the SMs that share an
//     instruction cache took up to 1.6 times as long as the ones that do not (128K tokens: 980 us for the slowest,
//     600 for the fastest; below 50 KB: 650 and 600).  Hence no division in the unit decoding, rolled loops in the
//     epilogue and for masked blocks, TMA stores, one instantiation per data type.
//
// Lists are walked from the last entry (the diagonal block when causal, which usually holds the row maximum) to the
// first, so the running maximum settles at the first block and O is rarely rescaled.
// TMEM columns: [0,128) S of stream 0, [128,256) S of stream 1, [256,384) O of stream 0, [384,512) O of stream 1.
#include <math.h>

#include <atomic>
#include <type_traits>

#include "attention_common.cuh"

namespace xb {

constexpr int kAttnThreads = 512;
constexpr int kAttnSmemTiles = kTile16 * 6;                   // Q0, Q1, then two slots of K, V
constexpr int kStageBytes = 4 * 2 * 32 * 128;                 // per epilogue warp: 32 rows x 2 x 64 16-bit columns
// A step of the K/V loader, published for the MMA issuer in a ring: which streams use the K/V pair, and whether it is the
// first / the last block of their tile
constexpr int kRingEntries = 8;
constexpr int kStepUses = 1, kStepFirst = 4, kStepLast = 16, kStepEnd = 64;      // << stream, except the last
// A unit, published by the K/V loader for the other roles: each stream's tile and its number of blocks
struct UnitTile {
  int b, h, qb, n;        // qb < 0: no tile; n < 0: no more units
};
constexpr int kUnitSlots = 4;
constexpr int kUnitReaders = 13;                              // warps that read it
constexpr int kAttnSmem = kAttnSmemTiles + kStageBytes + 2 * 2 * 128 * 4 /*row sums*/ + kRingEntries * 4 +
                          kUnitSlots * 2 * 16 + 16 + 512 /*barriers*/;
constexpr int kReuseBlocks = 8;           // lists up to that length may find a K/V tile of the unit before in its slot (longer: not worth the look)
constexpr float kRescaleThreshold = 8.0f;  // log2 units

struct Tile {
  int b, h, qb;      // qb < 0: no tile
};
__device__ __forceinline__ size_t tile_row(const AttnParams& p, const Tile& t) {
  return (static_cast<size_t>(t.b) * p.hq + t.h) * p.q_blocks + t.qb;
}
// Tile s of unit u.  With a tile list (kList, and one given): its entries 2u and 2u+1 (-1: none), tile i being (b, h, qb)
// with qb from the last to the first.  Otherwise a "super row" is two query blocks hi, hi-1; its hq units per batch entry
// are, for each kv head, the pairs of query heads at hi, then those at hi-1, and for an odd group first one unit that takes
// the last head at hi and hi-1.  Causal: super row by super row, the heaviest (last) first.  Non-causal: kv head by kv
// head, so that the CTAs work on one head's K and V at a time.
// kSplit: unit u is the tile of that number in a tile list, both streams'.
template <bool kList, bool kSplit = false>
__device__ __forceinline__ Tile unit_tile(const AttnParams& p, int u, int s) {
  Tile t;
  if constexpr (kSplit) {
    const int rest = fast_div(u, p.by_hq, t.h);
    t.qb = p.q_blocks - 1 - fast_div(rest, p.by_batch, t.b);
  } else if (kList && p.tile_list) {
    t.b = t.h = 0;
    t.qb = -1;
    const int i = 2 * u + s < p.list_tiles ? ld_written(p.tile_list + 2 * u + s) : -1;
    if (i < 0) return t;
    const int rest = fast_div(i, p.by_hq, t.h);
    t.qb = p.q_blocks - 1 - fast_div(rest, p.by_batch, t.b);
  } else {
    int x, j, g;
    const int hi = fast_div(u, p.by_units, x), lo = fast_div(x, p.by_group, j);
    const int r = p.causal ? hi : lo, bg = p.causal ? lo : hi;
    t.b = fast_div(bg, p.by_hkv, g);
    const int group = static_cast<int>(p.by_group.d), odd = group & 1, pairs = group >> 1;
    const int lower = j - odd >= pairs ? 1 : 0;
    const int across = odd && j == 0 ? 1 : 0;
    t.qb = p.q_blocks - 1 - 2 * r - (across ? s : lower);
    t.h = g * group + (across ? group - 1 : 2 * (j - odd - lower * pairs) + s);
  }
  return t;
}
// number of listed blocks; a dense call lists every block that holds a key the tile's last row may see
__device__ __forceinline__ int tile_count(const AttnParams& p, const int32_t* __restrict__ block_cnt, const Tile& t) {
  if (t.qb < 0) return 0;
  if (block_cnt) {
    const int n = ld_written(block_cnt + tile_row(p, t));
    return n < 0 ? 0 : (n < p.list_k_blocks ? n : p.list_k_blocks);      // (a list is read from its end: never past its row)
  }
  if (!p.causal) return p.list_k_blocks;
  int last = t.qb * 128 + 127;
  last = (last < p.q_len - 1 ? last : p.q_len - 1) + p.k_len - p.q_len;
  const int n = last / 128 + 1;
  return n < p.list_k_blocks ? n : p.list_k_blocks;
}
// Blocks of a tile of n that stream s walks (n < 0: no more units): all of them, or, split between the streams, every other one.
template <bool kSplit>
__device__ __forceinline__ int share(int n, int s) { return kSplit && n > 0 ? (n + 1 - s) >> 1 : n; }
// A tile's list as its walkers see it: walk position j maps to list[n - 1 - j] (split: list[n - 1 - s - 2 j]).
struct List {
  const int32_t* last;     // the first entry walked; null in a dense call
  int n, top;              // entries to walk; (split) place of the first one
};
template <bool kSplit>
__device__ __forceinline__ List tile_list(const AttnParams& p, const int32_t* __restrict__ block_idx, const Tile& t, int n, int s) {
  List l;
  l.top = kSplit ? n - 1 - s : 0;
  l.last = block_idx ? block_idx + tile_row(p, t) * p.list_k_blocks + (kSplit ? l.top : n - 1) : nullptr;
  l.n = share<kSplit>(n, s);
  return l;
}
// entry j of the list, walking order
template <bool kSplit>
__device__ __forceinline__ int list_entry(const List& l, int j) {
  if (j >= l.n) return 0;
  if (!l.last) return kSplit ? l.top - 2 * j : l.n - 1 - j;
  // (its volatile asm also pins the issue point: a plain load would be sunk by the compiler to its first use, which turns
  // the intended prefetch into an exposed memory latency)
  return ld_written(l.last - (kSplit ? 2 * j : j));
}

// Reader of the published units.
struct Units {
  const volatile UnitTile* ring;          // [slot][stream]
  uint32_t full, empty;                   // shared-memory addresses of the slots' barriers
  volatile int* abort_flag;
  uint32_t k;
  // whole warp: waits for the next unit; false after an abort
  __device__ __forceinline__ bool wait() {
    return __all_sync(0xffffffffu, mbar_wait(full + 8 * (k % kUnitSlots), (k / kUnitSlots) & 1, abort_flag));
  }
  __device__ __forceinline__ UnitTile tile(int s) const {
    const int4 v = *reinterpret_cast<const int4*>(const_cast<const UnitTile*>(ring) + 2 * (k % kUnitSlots) + s);
    UnitTile t;
    t.b = v.x; t.h = v.y; t.qb = v.z; t.n = v.w;
    return t;
  }
  __device__ __forceinline__ void release(int lane) {
    __syncwarp();
    if (lane == 0) mbar_arrive(empty + 8 * (k % kUnitSlots));
    ++k;
  }
};

// kBf16: bf16 or fp16 (a template parameter: as a run-time switch every packed pair cost both conversions and a select).
// kOutF32: the output is written as fp32.  kList: the units may come from a list.
// kTwo: a CTA takes two units next to one another at a time (the causal numbering, no list of units), see the loader.
// kSplit: a unit is a single tile, of whose list each stream walks every other block; the epilogue puts the two together.
template <bool kBf16, bool kOutF32, bool kList, bool kTwo, bool kSplit>
__global__ void __launch_bounds__(kAttnThreads, 1)
block_sparse_attn_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                         const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmO,
                         const AttnParams p_in,
                         const int32_t* __restrict__ block_idx, const int32_t* __restrict__ block_cnt,
                         const int32_t* __restrict__ rest_list, const int* __restrict__ pair_header,
                         int pair_min_share, int* status) {
  // The kernel is launched with 512 threads x 128 registers; setmaxnreg moves registers between warpgroups inside
  // that allocation.  A softmax thread keeps a row's 128 scores in registers; shared memory takes nearly the whole
  // L1, so a register spilled to local memory would cost an L2 round trip.
  constexpr int kRegSoftmax = 192, kRegEpilogue = 64, kRegLoadMma = 64;
  static_assert(8 * kRegSoftmax + 4 * kRegEpilogue + 4 * kRegLoadMma <= 16 * 128, "register budget of the roles");
  extern __shared__ __align__(1024) uint8_t smem[];
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);     // (uniform for the compiler too)
  const int lane = threadIdx.x & 31;
  if ((smem_u32(smem) & 1023u) != 0) {              // the swizzled tiles need 1024-byte alignment
    if (threadIdx.x == 0 && status) atomicExch(status, static_cast<int>(kDevBadSmemAlign));
    return;
  }
  uint8_t* stage_base = smem + kAttnSmemTiles;
  float* s_l = reinterpret_cast<float*>(stage_base + kStageBytes);                 // [stream][2][128] final row sums of two tiles (split: of one, and the maxima they are against)
  volatile int* ring = reinterpret_cast<volatile int*>(s_l + 2 * 2 * 128);         // [step]
  UnitTile* unit_ring = reinterpret_cast<UnitTile*>(s_l + 2 * 2 * 128 + kRingEntries);         // [slot][stream]
  uint8_t* answer = reinterpret_cast<uint8_t*>(unit_ring + 2 * kUnitSlots);                    // of the request for a unit
  uint64_t* bars = reinterpret_cast<uint64_t*>(answer + 16);
  // per slot: K_*, V_*; per stream: the others; then UNIT_FULL, UNIT_EMPTY per unit slot, and the answer's
  enum { K_FULL = 0, K_EMPTY, V_FULL, V_EMPTY, Q_FULL, Q_EMPTY, S_FULL, P_READY, O_FULL = P_READY + 2, O_EMPTY, NBAR };
  const uint32_t bar0 = smem_u32(bars);
  auto bar = [&](int s, int which) -> uint32_t { return bar0 + 8u * (NBAR * s + which); };
  const uint32_t unit_full = bar0 + 8u * (2 * NBAR), unit_empty = unit_full + 8u * kUnitSlots,
                 answer_full = unit_empty + 8u * kUnitSlots;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * NBAR + 2 * kUnitSlots + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
#ifdef XB_TRACE
  uint32_t trace_n = 0;
  const int trace_role = warp < 8 ? ((warp & 3) == 0 ? 2 + (warp >> 2) : 7 + 3 * (warp >> 2) + (warp & 3) - 1)
                                  : (warp < 12 ? 4 : (warp == 12 ? 0 : (warp == 13 ? 1 : (warp == 14 ? 5 : 6))));
#endif
  if (threadIdx.x == 0) {
#pragma unroll 1
    for (int s = 0; s < 2; ++s)
#pragma unroll 1
      for (int w = 0; w < NBAR; ++w)
        mbar_init(bar(s, w), (w == P_READY || w == P_READY + 1 || w == O_EMPTY) ? 128 : 1);
#pragma unroll 1
    for (int w = 0; w < kUnitSlots; ++w) {
      mbar_init(unit_full + 8u * w, 1);
      mbar_init(unit_empty + 8u * w, kUnitReaders);
    }
    mbar_init(answer_full, 1);
    *abort_flag = 0;
    fence_mbar_init();
    tma_prefetch_desc(&tmQ);
    tma_prefetch_desc(&tmK);
    tma_prefetch_desc(&tmV);
    tma_prefetch_desc(&tmO);
  }
  if (warp == 13) {
    tmem_alloc(smem_u32(tmem_slot), 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  // The kernel may have been launched while the one before it in the stream was still running: up to here it has
  // touched nothing that one writes.  With a pair kernel in front: the items it left (a list) if it ran, all items if
  // it declined.
  pdl_wait();
  AttnParams p = p_in;
  if (kList && rest_list && pair_path_chosen(pair_header, pair_min_share)) {
    p.tile_list = rest_list;
    p.list_tiles = *reinterpret_cast<const volatile int*>(pair_header + kPairRestCount);
  }
  // (units of the pass over a pair kernel's leavings, or of the whole call if it declined)
  const int rest_units = p.tile_list ? (p.list_tiles + 1) / 2 : (p.q_blocks + 1) / 2 * p.batch * p.hq;
  Units units;
  units.ring = unit_ring;
  units.full = unit_full;
  units.empty = unit_empty;
  units.abort_flag = abort_flag;
  units.k = 0;

  if (warp >= 12) {
    reg_set_from<kRegLoadMma, 128>();
    if (warp == 12) {
      // ------------------------------------------------------------ K/V loader: the union of the two lists
      // Lanes 0-15 walk the list of stream 0, lanes 16-31 that of stream 1, with a window of 16 entries each.
      const int s = lane >> 4, wl = lane & 15;
      uint32_t step = 0;
      bool ok = true;
      auto wait = [&](uint32_t b, uint32_t ph) -> bool { return __all_sync(0xffffffffu, mbar_wait(b, ph, abort_flag)); };
      Tile tn;
      List ln;                                          // the next unit's, with the first window
      int wn = 0, unit = kTwo ? 2 * blockIdx.x : blockIdx.x;
      bool second = false;                              // (kTwo) `unit` is the second one of its request
      uint32_t requests = 0;
      int held[2] = {-1, -1};                           // (kTwo) the K/V tiles in the two slots, numbered through batch and heads
      // The first turn of the loop has no lists to load, it only fetches those of the CTA's own unit; turn k works on the
      // CTA's unit k - 1 and requests and fetches unit k.  With two units per request (kTwo) the second one is the
      // other pair of heads at the same rows, whose list is mostly the same: of two blocks (sink and diagonal), say, both are still
      // in the slots where the second unit wants them, and are not loaded again.
      ln.n = 0;
      ln.last = nullptr;
      tn.b = tn.h = 0;
#pragma unroll 1
      for (uint32_t k = 0; unit >= 0 && ok; ++k) {
        const List l = ln;
        int i = 0, w = wn, g_;
        const int kvh = __shfl_sync(0xffffffffu, fast_div(tn.h, p.by_group, g_), 0), b = __shfl_sync(0xffffffffu, tn.b, 0);
        bool more = false, reuse = false;
        int tile0 = 0;
        if constexpr (kTwo) {
          more = k > 0 && !second && unit + 1 < rest_units;
          reuse = __all_sync(0xffffffffu, l.n <= kReuseBlocks);
          tile0 = (b * p.hkv + kvh) * p.list_k_blocks;
        }
        if (k > 0 && !more && lane == 0 && !(kList && rest_list)) {
          mbar_expect_tx(answer_full, 16);
          clc_try_cancel(smem_u32(answer), answer_full);
        }
        __syncwarp();
        int wx = list_entry<kSplit>(l, 16 + wl);
        bool fetched = false;
#pragma unroll 1
        while (true) {
          const bool have = i < l.n;
          if (__any_sync(0xffffffffu, have)) {
            const int c = __shfl_sync(0xffffffffu, w, (lane & 16) | (i & 15)), own = have ? c : -1;
            const int other = __shfl_xor_sync(0xffffffffu, own, 16), blk = own > other ? own : other;
            const bool f = have && own == blk;
            int e = f ? (kStepUses | (i == 0 ? kStepFirst : 0) | (i == l.n - 1 ? kStepLast : 0)) << s : 0;
            e |= __shfl_xor_sync(0xffffffffu, e, 16);
            const int sl = step & 1;
            const uint32_t ph = ((step >> 1) & 1) ^ 1, dst = smem_u32(smem + (2 + 2 * sl) * kTile16);
            bool there = false;
            if constexpr (kTwo) {
              if (reuse) there = (sl ? held[1] : held[0]) == tile0 + blk;
              if (sl) held[1] = tile0 + blk; else held[0] = tile0 + blk;
            }
            if (!wait(bar(sl, K_EMPTY), ph)) { ok = false; break; }
            if (lane == 0) {
              XB_TRACE_EV(0x12, step);
              ring[step & (kRingEntries - 1)] = e;
              if (kTwo && there) {
                mbar_arrive(bar(sl, K_FULL));
              } else {
                mbar_expect_tx(bar(sl, K_FULL), kTile16);
                tma_load_5d(dst, &tmK, bar(sl, K_FULL), 0, blk * 128, 0, kvh, b);
              }
            }
            if (!wait(bar(sl, V_EMPTY), ph)) { ok = false; break; }
            if (lane == 0) {
              XB_TRACE_EV(0x13, step);
              if (kTwo && there) {
                mbar_arrive(bar(sl, V_FULL));
              } else {
                mbar_expect_tx(bar(sl, V_FULL), kTile16);
                tma_load_5d(dst + kTile16, &tmV, bar(sl, V_FULL), 0, blk * 128, 0, kvh, b);
              }
            }
            ++step;
            if (f && (++i & 15) == 0) {
              w = wx;
              wx = list_entry<kSplit>(l, i + 16 + wl);
            }
            __syncwarp();
          } else if (fetched) {
            break;
          }
          if (!fetched) {
            // the next unit: published, its lists on their way while this unit's blocks are loaded
            fetched = true;
            if (kList && rest_list) {
              if (k > 0) unit += gridDim.x;
              if (unit >= rest_units) unit = -1;
            } else if (kTwo && more) {
              ++unit;
              second = true;
            } else if (k > 0) {
              if (!wait(answer_full, (kTwo ? requests : k - 1) & 1)) { ok = false; break; }
              unit = clc_answer(smem_u32(answer));
              if constexpr (kTwo) {
                if (unit > 0) unit *= 2;
                second = false;
                ++requests;
              }
              fence_proxy_async_smem();                 // read before the next answer is written
            }
            int count = -1;                             // of the tile's blocks (split: of both streams)
            ln.n = -1;
            if (unit >= 0) {
              tn = unit_tile<kList, kSplit>(p, unit, s);
              count = tile_count(p, block_cnt, tn);
              ln = tile_list<kSplit>(p, block_idx, tn, count, s);
              wn = list_entry<kSplit>(ln, wl);
            }
            if (!wait(unit_empty + 8 * (k % kUnitSlots), (k / kUnitSlots & 1) ^ 1)) { ok = false; break; }
            if (wl == 0) reinterpret_cast<int4*>(unit_ring)[2 * (k % kUnitSlots) + s] = make_int4(tn.b, tn.h, tn.qb, count);
            __syncwarp();
            if (lane == 0) mbar_arrive(unit_full + 8 * (k % kUnitSlots));
          }
        }
      }
      // (no unit is left for this SM, and its last one's tiles are on their way: the set-up of the kernel after this one may run under the tail)
      if (!kList && !kTwo && p.early_next) pdl_launch_dependents();
      // the end marker: a step that no stream uses
      if (lane == 0 && ok && mbar_wait(bar(step & 1, K_EMPTY), ((step >> 1) & 1) ^ 1, abort_flag)) {
        ring[step & (kRingEntries - 1)] = kStepEnd;
        mbar_arrive(bar(step & 1, K_FULL));
      }
    } else if (warp == 14) {
      // ------------------------------------------------------------ Q loader of both streams
      uint32_t m = 0;                                   // parity of the tiles so far, bit s: stream s
      bool ok = true;
#pragma unroll 1
      while (ok && units.wait()) {
        const UnitTile t0 = units.tile(0), t1 = units.tile(1);
        units.release(lane);
        if (t0.n < 0) break;
        // a stream has one Q buffer, so a tile's Q can only be loaded when the last S of the stream's tile before it is
        // done: both tiles of the unit are first pulled into L2, so that the loads do not wait on HBM
        if (lane == 0) {
          if (t0.n > 0) tma_prefetch_l2_5d(&tmQ, 0, t0.qb * 128, 0, t0.h, t0.b);
          if (!kSplit && t1.n > 0) tma_prefetch_l2_5d(&tmQ, 0, t1.qb * 128, 0, t1.h, t1.b);
        }
        __syncwarp();
#pragma unroll 1
        for (int s = 0; s < 2; ++s) {
          const UnitTile t = s ? t1 : t0;
          if (share<kSplit>(t.n, s) == 0) continue;
          if (!__all_sync(0xffffffffu, mbar_wait(bar(s, Q_EMPTY), (m >> s & 1) ^ 1, abort_flag))) { ok = false; break; }
          if (lane == 0) {
            XB_TRACE_EV(0x10 + s, m);
            mbar_expect_tx(bar(s, Q_FULL), kTile16);
            tma_load_5d(smem_u32(smem + s * kTile16), &tmQ, bar(s, Q_FULL), 0, t.qb * 128, 0, t.h, t.b);
          }
          __syncwarp();
          m ^= 1u << s;
        }
      }
    } else if (warp == 13) {
      // ---------------------------------------------------------------- MMA issuer (converged warp, one thread issues: see
      // mma_ss_lead)
      constexpr uint32_t idesc_qk = make_idesc_f16(128, 128, kBf16, false, false);
      constexpr uint32_t idesc_pv = make_idesc_f16(128, 128, kBf16, false, true);
      const uint32_t lead = elect_one() ? 1u : 0u;
      // K-major operands, k-step k: 16 columns = 32 B inside the 64-column half (k & 3), the second half 16 KiB on;
      // V as MN-major operand: 16 keys per step = 16 x 128 B rows, the second 64 columns 16 KiB on
      const uint64_t dq0 = smem_desc_sw128(smem_u32(smem), 16, 1024);
      const uint64_t dk0 = smem_desc_sw128(smem_u32(smem + 2 * kTile16), 16, 1024);
      const uint64_t dv0 = smem_desc_sw128(smem_u32(smem + 3 * kTile16), kHalf16, 1024);
      auto wait = [&](uint32_t b, uint32_t ph) -> bool { return __all_sync(0xffffffffu, mbar_wait(b, ph, abort_flag)); };
      // S of stream s = Q K^T with the K tile of slot sl
      auto issue_qk = [&](int s, int sl) {
        const uint64_t dq = dq0 + static_cast<uint64_t>(s * (kTile16 >> 4));
        const uint64_t dk = dk0 + static_cast<uint64_t>(sl * ((2 * kTile16) >> 4));
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const uint32_t o = ((k >> 2) * kHalf16 + (k & 3) * 32) >> 4;
          mma_ss_lead(tmem_base + s * 128, dq + o, dk + o, idesc_qk, k > 0 ? 1u : 0u, lead);
        }
      };
      // O of stream s (+)= P V over keys 64 h .. 64 h + 63 of the V tile of slot sl
      auto issue_pv = [&](int s, int sl, int h, uint32_t accumulate) {
        const uint64_t dv = dv0 + static_cast<uint64_t>(sl * ((2 * kTile16) >> 4));
#pragma unroll
        for (int k = 0; k < 4; ++k)
          mma_ts_lead(tmem_base + 256 + s * 128, tmem_base + s * 128 + (4 * h + k) * 8, dv + (((4 * h + k) * 2048) >> 4),
                      idesc_pv, k > 0 ? 1u : accumulate, lead);
      };
      // One bit per stream: pend, its block of step u - 1 has its P.V outstanding; todo, step u's K is outstanding; next, it
      // has a block in step u.  In the fields of `st`: that block is the first / the last of its tile; parity of the
      // stream's blocks and of its tiles.
      constexpr int kFirst = 0, kLast = 2, kBlocks = 4, kTiles = 6;
      uint32_t st = 0, u = 0, pend = 0, todo = 3, next = 0;
      bool ok = true, have = false, v_used = false;     // have: the step's K is there and `e` is its entry
      int e = 0;
#pragma unroll 1
      while (ok) {
        const int sl = u & 1;
        // Without K a stream's outstanding P.V is issued all the same: the block may be the last one for a while, and the
        // next unit may even depend on it (its publication on the epilogue of this one).  So K is asked for before and
        // after each stream's P.V, and waited for only when neither stream has one left.
        auto look = [&](bool block) -> bool {
          if (!have) {
            have = block ? wait(bar(sl, K_FULL), (u >> 1) & 1)
                         : __all_sync(0xffffffffu, mbar_test(bar(sl, K_FULL), (u >> 1) & 1));
            if (have) e = __shfl_sync(0xffffffffu, ring[u & (kRingEntries - 1)], 0);
          }
          return have;
        };
        if (!look(pend == 0) && pend == 0) break;
        // (first the stream that can start on this step at once, its last block being done, if the other cannot)
        const int s0 = pend == 1 && have && (e & (kStepUses << 1)) ? 1 : 0;
#pragma unroll 1
        for (int i = 0; i < 2; ++i) {
          const int s = s0 ^ i;
          auto bit = [&](int field) -> uint32_t { return st >> (field + s) & 1u; };
          if (pend >> s & 1) {
            // P.V of the block of step u - 1, in two steps: keys 0-63 as soon as their half of P is written, so that
            // this half runs while the softmax warpgroup still exponentiates keys 64-127
            const uint32_t par = bit(kBlocks);
            if (!wait(bar(sl ^ 1, V_FULL), ((u - 1) >> 1) & 1)) { ok = false; break; }
            if (bit(kFirst) && !wait(bar(s, O_EMPTY), bit(kTiles) ^ 1)) { ok = false; break; }
            if (!wait(bar(s, P_READY), par)) { ok = false; break; }
            tc_fence_after();
            if (lead) XB_TRACE_EV(0x22 + 0x100 * s, u - 1);
            issue_pv(s, sl ^ 1, 0, bit(kFirst) ^ 1u);
            if (!wait(bar(s, P_READY + 1), par)) { ok = false; break; }
            tc_fence_after();
            if (lead) XB_TRACE_EV(0x25 + 0x100 * s, u - 1);
            issue_pv(s, sl ^ 1, 1, 1u);
            if (bit(kLast)) {
              mma_commit_lead(bar(s, O_FULL), lead);
              st ^= 1u << (kTiles + s);
            }
            st ^= 1u << (kBlocks + s);
            st &= ~((1u << kFirst | 1u << kLast) << s);
            pend &= ~(1u << s);
          }
          if (v_used && pend == 0) {
            mma_commit_lead(bar(sl ^ 1, V_EMPTY), lead);
            v_used = false;
          }
          if (!(todo >> s & 1) || !look(false)) continue;
          todo &= ~(1u << s);
          if (e >> s & kStepUses) {
            if (e >> s & kStepFirst) {
              if (!wait(bar(s, Q_FULL), bit(kTiles))) { ok = false; break; }
              st |= 1u << (kFirst + s);
            }
            tc_fence_after();
            if (lead) XB_TRACE_EV(0x20 + 0x100 * s, u);
            issue_qk(s, sl);
            mma_commit_lead(bar(s, S_FULL), lead);
            if (e >> s & kStepLast) {
              mma_commit_lead(bar(s, Q_EMPTY), lead);
              st |= 1u << (kLast + s);
            }
            next |= 1u << s;
          }
        }
        if (todo) continue;                             // K was not there for both
        if (e & kStepEnd) break;
        mma_commit_lead(bar(sl, K_EMPTY), lead);
        pend = next;
        next = 0;
        todo = 3;
        have = false;
        v_used = true;
        ++u;
      }
    }
  } else if (warp < 8) {
    // -------------------------------------------------------------------- softmax of stream (warp >> 2)
    reg_set_from<kRegSoftmax, 128>();
    const int s = warp >> 2;
    const int quad = warp & 3;
    const int r = quad * 32 + lane;
    const uint32_t lane_bits = static_cast<uint32_t>(quad * 32) << 16;
    const uint32_t ts = tmem_base + s * 128 + lane_bits;          // S / P of this stream, this row
    const uint32_t tmem_o = tmem_base + 256 + s * 128 + lane_bits;
    const int k_off = p.k_len - p.q_len;
    const unsigned long long scale2 = pack_f32x2(p.scale_log2, p.scale_log2);
    uint32_t bc = 0;
    bool ok = true;
    // the stream's tile in the next unit, with its list's first window on its way from memory.  (One unit at a time: to
    // wait here for a unit that lists anything would hold up the unit at hand, and with it the publication of the next.)
    UnitTile nt;
    int nwin = 0;
    auto list_of = [&](const UnitTile& ut) -> List {
      Tile tt;
      tt.b = ut.b; tt.h = ut.h; tt.qb = ut.qb;
      return tile_list<kSplit>(p, block_idx, tt, ut.n, s);
    };
    auto fetch = [&]() {
      if (!units.wait()) {
        nt.n = -1;
        return;
      }
      nt = units.tile(s);
      units.release(lane);
      if (nt.n > 0) nwin = list_entry<kSplit>(list_of(nt), lane);
    };
    int m = 0;
    nt.n = 0;
#pragma unroll 1
    while (ok && nt.n >= 0) {
      if (share<kSplit>(nt.n, s) == 0) {                // (at the start, too)
        fetch();
        continue;
      }
      const UnitTile t = nt;
      const List list = list_of(t);
      if (lane == 0) XB_TRACE_EV(0x36, m);
      const int n = list.n;
      const int q_pos = t.qb * 128 + r;
      int row_last = p.k_len - 1;                       // last key position this row may see
      if (p.causal && q_pos + k_off < row_last) row_last = q_pos + k_off;
      int row_last_lo = p.k_len - 1;                    // the same for the first row of the warp
      if (p.causal && t.qb * 128 + quad * 32 + k_off < row_last_lo) row_last_lo = t.qb * 128 + quad * 32 + k_off;
      float m_used = -INFINITY, l = 0.f;
      int w = nwin, w_next = list_entry<kSplit>(list, 32 + lane);
#pragma unroll 1
      for (int j = 0; j < n; ++j, ++bc) {
        if (j > 0 && (j & 31) == 0) {
          w = w_next;
          w_next = list_entry<kSplit>(list, j + 32 + lane);
        }
        const int k0 = __shfl_sync(0xffffffffu, w, j & 31) * 128;
        if (lane == 0) XB_TRACE_EV(0x30, bc);
        // waits are made warp-uniform: the tensor-memory loads/stores below are warp-collective
        if (!__all_sync(0xffffffffu, mbar_wait(bar(s, S_FULL), bc & 1, abort_flag))) { ok = false; break; }
        tc_fence_after();
        if (lane == 0) XB_TRACE_EV(0x31, bc);
        float mx8[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) mx8[q] = -INFINITY;
        auto chunk_max = [&](const uint32_t (&x)[32]) {
#pragma unroll
          for (int k = 0; k < 16; ++k)
            mx8[k & 7] = max3(mx8[k & 7], __uint_as_float(x[2 * k]), __uint_as_float(x[2 * k + 1]));
        };
        unsigned long long ls2[4], nmref2 = 0ull;
#pragma unroll
        for (int q = 0; q < 4; ++q) ls2[q] = 0ull;     // (+0.f, +0.f)
        // exp2 of 32 scores, their sum, and P packed to 16 bit
        auto chunk_exp = [&](const uint32_t (&x)[32], uint32_t (&pk)[16]) {
#pragma unroll
          for (int k = 0; k < 16; ++k) {
            float y0, y1;
            unpack_f32x2(fma_f32x2(pack_f32x2(__uint_as_float(x[2 * k]), __uint_as_float(x[2 * k + 1])), scale2, nmref2),
                         y0, y1);
            const float p0 = fast_exp2(y0), p1 = fast_exp2(y1);
            ls2[k & 3] = add_f32x2(ls2[k & 3], pack_f32x2(p0, p1));
            pk[k] = pack16t<kBf16>(p0, p1);
          }
        };
        // the running maximum moves to cover this block (lazily); O is rescaled if it holds anything already
        auto rescale = [&]() {
          const float mx = fmaxf(max3(mx8[0], mx8[1], mx8[2]), max3(max3(mx8[3], mx8[4], mx8[5]), mx8[6], mx8[7]));
          const float m_new = fmaxf(m_used, mx * p.scale_log2);
          const bool need = m_new > m_used + kRescaleThreshold || j == 0 || (m_used == -INFINITY && m_new > -INFINITY);
          if (__any_sync(0xffffffffu, need)) {
            const float alpha = !need ? 1.f : (m_used == -INFINITY ? 0.f : fast_exp2(m_used - m_new));
            if (j > 0) {
              // O may be touched: S of this block is complete, and its MMAs were issued after the stream's P.V of all
              // earlier blocks
              if (lane == 0) XB_TRACE_EV(0x32, bc);
#pragma unroll 1
              for (int c4 = 0; c4 < 8; ++c4) {
                uint32_t o[16];
                tmem_ld16(tmem_o + c4 * 16, o);
                tc_wait_ld();
#pragma unroll
                for (int k = 0; k < 16; ++k) o[k] = __float_as_uint(__uint_as_float(o[k]) * alpha);
                tmem_st16(tmem_o + c4 * 16, o);
              }
            }
            l *= alpha;
            if (need) m_used = m_new;
          }
          const float m_ref = m_used == -INFINITY ? 0.f : m_used;
          nmref2 = pack_f32x2(-m_ref, -m_ref);
          if (lane == 0) XB_TRACE_EV(0x35, bc);
        };
        // P of chunk c (32 keys, 16 packed columns) goes to columns [16 c, 16 c + 16): scores that have been read by now
        auto half_ready = [&](int h) {
          tc_wait_st();
          tc_fence_before();
          mbar_arrive(bar(s, P_READY + h));
        };
        // last visible column of the warp's first row: every row of the warp sees the whole block, or some do not
        const int lim_lo = row_last_lo - k0;
        if (lim_lo < 127) {
          // Some columns are hidden from some rows (diagonal blocks, the ragged last block): their scores are replaced by
          // -inf in tensor memory, in a rolled loop over the chunks concerned, because the code has to stay small.
          const int lim = row_last - k0;                // columns c <= lim are visible
#pragma unroll 1
          for (int c = lim_lo < 0 ? 0 : (lim_lo + 1) >> 5; c < 4; ++c) {
            uint32_t x[32];
            tmem_ld32(ts + c * 32, x);
            tc_wait_ld();
            const int lc = lim - 32 * c;
#pragma unroll
            for (int k = 0; k < 32; ++k) x[k] = k <= lc ? x[k] : 0xff800000u;
            tmem_st32(ts + c * 32, x);
          }
          tc_wait_st();
        }
        // (the diagonal block for its first 64 rows: no row of the warp sees keys 64-127)
        const bool upper_hidden = lim_lo < 33 && __shfl_sync(0xffffffffu, row_last - k0, 31) < 64;
        uint32_t v[4][32];
        tmem_ld32(ts, v[0]);
        tmem_ld32(ts + 32, v[1]);
        tc_wait_ld();
        tmem_ld32(ts + 64, v[2]);
        tmem_ld32(ts + 96, v[3]);
        chunk_max(v[0]);
        chunk_max(v[1]);
        tc_wait_ld();
        chunk_max(v[2]);
        chunk_max(v[3]);
        rescale();
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          uint32_t pk[16];
          chunk_exp(v[c], pk);
          tmem_st16(ts + c * 16, pk);
        }
        half_ready(0);
        if (lane == 0) XB_TRACE_EV(0x34, bc);
        if (upper_hidden) {
          uint32_t z[16];
#pragma unroll
          for (int k = 0; k < 16; ++k) z[k] = 0u;
          tmem_st16(ts + 32, z);
          tmem_st16(ts + 48, z);
        } else {
#pragma unroll
          for (int c = 2; c < 4; ++c) {
            uint32_t pk[16];
            chunk_exp(v[c], pk);
            tmem_st16(ts + c * 16, pk);
          }
        }
        {
          float a0, a1;
          unpack_f32x2(add_f32x2(add_f32x2(ls2[0], ls2[1]), add_f32x2(ls2[2], ls2[3])), a0, a1);
          l += a0 + a1;
        }
        if (j == n - 1) {                               // read by the epilogue once this tile's last P.V is done
          if constexpr (kSplit) {
            // (the epilogue may still be waiting for the other stream's part of the tile before)
            if (!__all_sync(0xffffffffu, mbar_wait(bar(s, O_EMPTY), (m & 1) ^ 1, abort_flag))) { ok = false; break; }
            s_l[s * 2 * 128 + r] = l;
            s_l[(s * 2 + 1) * 128 + r] = m_used;
          } else {
            s_l[(s * 2 + (m & 1)) * 128 + r] = l;
          }
        }
        half_ready(1);
        if (j == 0) fetch();
        if (lane == 0) XB_TRACE_EV(0x33, bc);
      }
      ++m;
    }
  } else {
    // -------------------------------------------------------------------- epilogue (warps 8-11), both streams
    reg_set_from<kRegEpilogue, 128>();
    const int quad = warp & 3;
    const int r = quad * 32 + lane;
    const uint32_t lane_bits = static_cast<uint32_t>(quad * 32) << 16;
    // A warp's 32 rows x 128 columns go, scaled and packed to 16 bit, to a staging tile of two 64-column halves in the
    // 128-byte swizzle pattern (16-byte chunk c of row r at chunk c ^ (r & 7)) and leave as two TMA stores, which also
    // clip the rows past q_len.  O leaves tensor memory before the stores, so that the stream's next tile can start
    // accumulating while this one is still being stored.
    uint8_t* stg = stage_base + quad * (2 * 32 * 128);
    uint32_t done = 0;                 // tiles with a list so far, mod 2: stream 0 in bit 0, stream 1 in bit 1
    bool ok = true;
    UnitTile t1;
#pragma unroll 1
    for (int i = 0; ok; ++i) {
      const int s = kSplit ? 0 : i & 1;
      UnitTile t = t1;
      if (s == 0) {
        if (!units.wait()) break;
        t = units.tile(0);
        t1 = units.tile(1);
        units.release(lane);
      }
      const int n = t.n;
      if (n < 0) break;
      if (t.qb < 0) continue;
      float inv = 0.f, inv1 = 0.f;                      // what O is multiplied with; split: and the other stream's
      if constexpr (kSplit) {
#pragma unroll 1
        for (int x = 0; x < 2 && x < n && ok; ++x) {
          ok = __all_sync(0xffffffffu, mbar_wait(bar(x, O_FULL), (done >> x) & 1, abort_flag));
          done ^= 1u << x;
        }
        if (!ok) break;
        tc_fence_after();
        if (n > 0) {
          // the two halves of the row against the larger of their maxima
          const float l0 = s_l[r], m0 = s_l[128 + r], l1 = n > 1 ? s_l[2 * 128 + r] : 0.f, m1 = n > 1 ? s_l[3 * 128 + r] : -INFINITY;
          const float top = fmaxf(m0, m1);
          const float a0 = m0 == -INFINITY ? 0.f : fast_exp2(m0 - top), a1 = m1 == -INFINITY ? 0.f : fast_exp2(m1 - top);
          const float sum = l0 * a0 + l1 * a1, over = sum > 0.f ? 1.f / sum : 0.f;
          inv = a0 * over;
          inv1 = a1 * over;
        }
      } else if (n > 0) {
        const uint32_t m = (done >> s) & 1;
        done ^= 1u << s;
        if (threadIdx.x == 256) XB_TRACE_EV(0x40 + s, m);
        if (!__all_sync(0xffffffffu, mbar_wait(bar(s, O_FULL), m, abort_flag))) { ok = false; break; }
        tc_fence_after();
        if (threadIdx.x == 256) XB_TRACE_EV(0x42 + s, m);
        const float l = s_l[(s * 2 + m) * 128 + r];
        inv = l > 0.f ? 1.f / l : 0.f;
      }
      const uint32_t tmem_o = tmem_base + 256 + s * 128 + lane_bits;
      // 32 columns of O from `c` on, scaled (split: the two streams' parts added), as words
      auto load_out = [&](int c, uint32_t (&v)[32]) {
        tmem_ld32(tmem_o + c, v);
        tc_wait_ld();
#pragma unroll
        for (int k = 0; k < 32; ++k) v[k] = __float_as_uint(__uint_as_float(v[k]) * inv);
        if constexpr (kSplit) {
          if (n > 1) {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              uint32_t y[16];
              tmem_ld16(tmem_o + 128 + c + 16 * h, y);
              tc_wait_ld();
#pragma unroll
              for (int k = 0; k < 16; ++k) v[16 * h + k] = __float_as_uint(__uint_as_float(v[16 * h + k]) + __uint_as_float(y[k]) * inv1);
            }
          }
        }
      };
      auto o_read = [&]() {
        if (n > 0) {
          tc_fence_before();
          mbar_arrive(bar(s, O_EMPTY));
          if (kSplit && n > 1) mbar_arrive(bar(1, O_EMPTY));
        }
      };
      if constexpr (kOutF32) {
        const int q_row0 = t.qb * 128 + quad * 32;      // first row of this warp
        // 32 columns at a time through the two halves of the staging tile in turn
#pragma unroll 1
        for (int c = 0; c < 4; ++c) {
          uint32_t v[32];
          if (n > 0) {
            load_out(c * 32, v);
          } else {                                      // an empty list: zeros
#pragma unroll
            for (int k = 0; k < 32; ++k) v[k] = 0u;
          }
          if (lane == 0) tma_store_wait_read_1();       // the half's previous store has read it
          __syncwarp();
          uint8_t* half = stg + (c & 1) * (32 * 128);
#pragma unroll
          for (int q4 = 0; q4 < 8; ++q4)
            *reinterpret_cast<uint4*>(half + lane * 128 + ((q4 ^ (lane & 7)) << 4)) =
                make_uint4(v[4 * q4], v[4 * q4 + 1], v[4 * q4 + 2], v[4 * q4 + 3]);
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) {
            if (q_row0 < p.q_len) tma_store_5d(&tmO, smem_u32(half), 0, q_row0, c, t.h, t.b);
            tma_store_commit();
          }
        }
        o_read();
      } else {
        if (lane == 0) tma_store_wait_read();           // the staging tile's previous stores have read it
        __syncwarp();
#pragma unroll 1
        for (int c = 0; c < 4; ++c) {
          uint32_t pk[16];
          if (n > 0) {
            uint32_t v[32];
            load_out(c * 32, v);
#pragma unroll
            for (int k = 0; k < 16; ++k) pk[k] = pack16t<kBf16>(__uint_as_float(v[2 * k]), __uint_as_float(v[2 * k + 1]));
          } else {                                      // an empty list: zeros
#pragma unroll
            for (int k = 0; k < 16; ++k) pk[k] = 0u;
          }
          uint8_t* row = stg + (c >> 1) * (32 * 128) + lane * 128;
#pragma unroll
          for (int q4 = 0; q4 < 4; ++q4)
            *reinterpret_cast<uint4*>(row + (((((c & 1) << 2) | q4) ^ (lane & 7)) << 4)) =
                make_uint4(pk[4 * q4], pk[4 * q4 + 1], pk[4 * q4 + 2], pk[4 * q4 + 3]);
        }
        o_read();
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) {
          const int q_row0 = t.qb * 128 + quad * 32;    // first row of this warp
          if (q_row0 < p.q_len) {
            tma_store_5d(&tmO, smem_u32(stg), 0, q_row0, 0, t.h, t.b);
            tma_store_5d(&tmO, smem_u32(stg + 32 * 128), 0, q_row0, 1, t.h, t.b);
            tma_store_commit();
          }
        }
      }
      if (threadIdx.x == 256) XB_TRACE_EV(0x44 + s, 0);
    }
    if (lane == 0) tma_store_wait_all();                // the staging tiles must outlive the stores that read them
  }

  // -------------------------------------------------------------------- teardown
  tc_fence_before();
  __syncthreads();
  if (*abort_flag) {
    const long long t0 = clock64();
    while (clock64() - t0 < 2000000) { __nanosleep(1000); }
    if (threadIdx.x == 0 && status) atomicExch(status, static_cast<int>(kDevWaitTimeout));
    __syncthreads();
  }
  if (warp == 13) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

// ------------------------------------------------------------------------------------------------ unit order
// Non-causal masks have no order of their own (video diffusion: rows list 5 to 891 of 931 blocks, anywhere in the
// sequence).  The units are put in this order: first the very long ones of all heads, then kv head by kv head the others,
// longest first.  Two effects:
//  * the CTAs work on one kv head at a time, so the K/V tiles they gather come from that head's tensors only -- 61 MB at
//    119K tokens, which stay in L2, where a walk over all 24 heads at once (1.46 GB) re-reads every tile from HBM;
//  * a unit that would keep a CTA busy for a good part of the whole call (the rows of the text tokens list nearly every
//    block) starts at once instead of near the end.
// One CTA per (batch, kv head) sorts that head's units with a counting sort by the two tiles' list lengths (sums above
// kOrderBuckets - 1 share the first bucket; the order inside a bucket is as the atomics fall, which changes nothing in
// the result) and counts the very long units of all heads by itself, so that the CTAs need not wait for one another.
constexpr int kOrderBuckets = 4096;
constexpr int kOrderThreads = 1024;
__global__ void __launch_bounds__(kOrderThreads, 1)
attn_order_kernel(const AttnParams p, const int32_t* __restrict__ block_cnt, int sms, int32_t* __restrict__ sorted) {
  __shared__ int hist[kOrderBuckets];
  __shared__ int warp_sum[kOrderThreads / 32];
  __shared__ unsigned long long s_blocks[kOrderThreads / 32];
  __shared__ int s_long[3];           // very long units: of all heads, of the heads before this one, of this one
  pdl_launch_dependents();            // the attention kernel may take its place; it waits for this grid to end
  pdl_wait();
  const int tid = threadIdx.x;
  const int n_seg = static_cast<int>(p.by_units.d);                      // units of a (batch, kv head)
  const int n_heads = gridDim.x, first = blockIdx.x * n_seg;
  if (tid < 3) s_long[tid] = 0;
  for (int i = tid; i < kOrderBuckets; i += kOrderThreads) hist[i] = 0;
  __syncthreads();
  // blocks listed by the whole call; a unit with more than an eighth of one SM's share of them is a very long one
  const int rows = p.batch * p.hq * p.q_blocks;
  unsigned long long sum = 0;
#pragma unroll 4
  for (int i = tid; i < rows; i += kOrderThreads) sum += static_cast<unsigned>(ld_written(block_cnt + i));
  // (Warp by warp: an atomic addition of 64 bits in shared memory is a loop, and with all threads' going to one word this kernel took
  // 47 us for 24 heads of 250 query blocks and 62 for 930; now 7 and 15.)
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
  if ((tid & 31) == 0) s_blocks[tid >> 5] = sum;
  __syncthreads();
  sum = 0;
#pragma unroll
  for (int w = 0; w < kOrderThreads / 32; ++w) sum += s_blocks[w];
  unsigned long long lim64 = sum / (8ull * sms);
  const int limit = lim64 < 64 ? 64 : (lim64 > kOrderBuckets - 2 ? kOrderBuckets - 2 : static_cast<int>(lim64));
  auto length = [&](int u) {
    const Tile t0 = unit_tile<false>(p, u, 0), t1 = unit_tile<false>(p, u, 1);
    const int c = tile_count(p, block_cnt, t0) + tile_count(p, block_cnt, t1);
    return c < 0 ? 0 : (c > kOrderBuckets - 1 ? kOrderBuckets - 1 : c);
  };
  for (int u = tid; u < n_heads * n_seg; u += kOrderThreads) {
    const int c = length(u);
    const bool own = u >= first && u < first + n_seg;
    if (own) atomicAdd(&hist[kOrderBuckets - 1 - c], 1);                 // the bucket index grows as the lists get shorter
    if (c > limit) {
      atomicAdd(&s_long[0], 1);
      if (own) atomicAdd(&s_long[2], 1);
      else if (u < first) atomicAdd(&s_long[1], 1);
    }
  }
  __syncthreads();
  // exclusive prefix over the buckets, four per thread
  int h[4], hsum = 0;
#pragma unroll
  for (int q = 0; q < 4; ++q) { h[q] = hsum; hsum += hist[4 * tid + q]; }
  int incl = hsum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, incl, o);
    if ((tid & 31) >= o) incl += v;
  }
  if ((tid & 31) == 31) warp_sum[tid >> 5] = incl;
  __syncthreads();
  if (tid < 32) {
    int w = warp_sum[tid];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, w, o);
      if (tid >= o) w += v;
    }
    warp_sum[tid] = w;                 // inclusive over the warps
  }
  __syncthreads();
  const int base = ((tid >> 5) > 0 ? warp_sum[(tid >> 5) - 1] : 0) + incl - hsum;
#pragma unroll
  for (int q = 0; q < 4; ++q) hist[4 * tid + q] = base + h[q];           // from here on: the bucket's next free place
  __syncthreads();
  const int all_long = s_long[0], before = s_long[1], own_long = s_long[2];
  for (int u = first + tid; u < first + n_seg; u += kOrderThreads) {
    const int rank = atomicAdd(&hist[kOrderBuckets - 1 - length(u)], 1);
    const int at = rank < own_long ? before + rank : all_long + first - before + (rank - own_long);
    const Tile t0 = unit_tile<false>(p, u, 0), t1 = unit_tile<false>(p, u, 1);
    // the numbering of the tile list: ((q_blocks - 1 - qb) * batch + b) * hq + h
    auto item = [&](const Tile& t) { return t.qb < 0 ? -1 : ((p.q_blocks - 1 - t.qb) * p.batch + t.b) * p.hq + t.h; };
    sorted[2 * at] = item(t0);
    sorted[2 * at + 1] = item(t1);
  }
}

size_t order_workspace_bytes(int batch, int hq, int q_len) {
  return static_cast<size_t>(batch) * hq * (((static_cast<size_t>(q_len) + 127) / 128 + 1) / 2) * 2 * sizeof(int32_t);
}

size_t pair_workspace_bytes(int batch, int hq, int hkv, int q_len);
bool pair_path_applies(int hq, int hkv, int k_len);
int block_sparse_attn_pair_launch(const CUtensorMap& tmQ, const CUtensorMap& tmKf, const CUtensorMap& tmVf,
                                  const AttnParams& p, const int32_t* block_idx, const int32_t* block_cnt, void* out,
                                  void* workspace, size_t workspace_bytes, const int32_t** rest_list,
                                  const int** header, int min_share_pct, int* status, cudaStream_t stream);

// Share (per cent) of a call's listed blocks that must qualify for the pair kernel before the call is split; a
// process-wide setting, read when a call is enqueued.  0: split whenever anything qualifies; > 100: never.
static std::atomic<int> g_pair_min_share{kPairMinSharePct};
int pair_min_share_pct(int set_to) {
  return set_to < 0 ? g_pair_min_share.load() : g_pair_min_share.exchange(set_to);
}

size_t block_sparse_attn_workspace_bytes(int batch, int hq, int hkv, int q_len, int k_len) {
  if (batch < 1 || hq < 1 || hkv < 1 || hq % hkv != 0 || q_len < 1 || k_len < 1) return 0;
  const size_t order = order_workspace_bytes(batch, hq, q_len);
  const size_t pair = pair_path_applies(hq, hkv, k_len) ? pair_workspace_bytes(batch, hq, hkv, q_len) : 0;
  return pair > order ? pair : order;
}

// Without lists (block_idx and block_cnt null) the call is dense.  With a workspace a causal call (with an even number >= 2
// of query heads per kv head) runs in two parts: the group items whose heads all list the same one or two blocks go to the
// pair kernel (attention_pair.cu), everything else to the general kernel, which takes its tiles from the list the pair
// path leaves (a group's query heads stand next to one another in it, so two entries read the same kv head).  A
// non-causal call with a workspace has its units ordered first (attn_order_kernel).
int block_sparse_attn_launch(const void* q, const void* k, const void* v, int dtype, int batch, int hq, int hkv,
                             int q_len, int k_len, int head_dim, int64_t qsb, int64_t qsh, int64_t qsl, int64_t ksb,
                             int64_t ksh, int64_t ksl, int64_t vsb, int64_t vsh, int64_t vsl,
                             const int32_t* block_idx, const int32_t* block_cnt, int causal, float scale, void* out,
                             int64_t osb, int64_t osh, int64_t osl, void* workspace, size_t workspace_bytes, int max_list,
                             int* status, cudaStream_t stream) {
  if (!q || !k || !v || !out || (block_idx == nullptr) != (block_cnt == nullptr)) return XATTN_B200_ERR_ARG;
  const bool dense = block_idx == nullptr;
  if (dtype != XATTN_B200_BF16 && dtype != XATTN_B200_F16 && dtype != XATTN_B200_BF16_OUT_F32) return XATTN_B200_ERR_ARG;
  const bool out_f32 = dtype == XATTN_B200_BF16_OUT_F32;
  if (head_dim != 128 || batch < 1 || hq < 1 || hkv < 1 || hq % hkv != 0 || q_len < 1 || k_len < 1)
    return XATTN_B200_ERR_ARG;
  if (causal && k_len < q_len) return XATTN_B200_ERR_ARG;
  if ((reinterpret_cast<uintptr_t>(out) & 15) || (osl % (out_f32 ? 4 : 8)) || (osh % (out_f32 ? 4 : 8)) || (osb % (out_f32 ? 4 : 8))) return XATTN_B200_ERR_ARG;
  if (!(scale > 0.f)) return XATTN_B200_ERR_ARG;
  int rc;
  if ((rc = check_sm100())) return rc;
  CUtensorMap tmQ, tmK, tmV, tmO;
  if ((rc = make_qkv_map(&tmQ, q, q_len, hq, batch, qsb, qsh, qsl, 128))) return rc;
  if ((rc = make_qkv_map(&tmK, k, k_len, hkv, batch, ksb, ksh, ksl, 128))) return rc;
  if ((rc = make_qkv_map(&tmV, v, k_len, hkv, batch, vsb, vsh, vsl, 128))) return rc;
  // the output: a store box is 32 rows of 128 bytes, one of two (fp32: four) column parts
  if ((rc = make_rows_map(&tmO, out, q_len, hq, batch, osb, osh, osl, 32, 1, out_f32 ? 4 : 2))) return rc;
  AttnParams p;
  p.batch = batch; p.hq = hq; p.hkv = hkv; p.q_len = q_len; p.k_len = k_len;
  p.q_blocks = (q_len + 127) / 128; p.list_k_blocks = (k_len + 127) / 128;
  p.causal = causal ? 1 : 0; p.is_bf16 = dtype != XATTN_B200_F16 ? 1 : 0;
  p.scale_log2 = scale * 1.4426950408889634f;
  p.osb = osb; p.osh = osh; p.osl = osl;
  p.tile_list = nullptr;
  p.list_tiles = 0;
  p.early_next = 0;
  const int super_rows = (p.q_blocks + 1) / 2;
  const long long units = static_cast<long long>(super_rows) * batch * hq;
  if (units > 0x3fffffffLL || p.list_k_blocks > 65534) return XATTN_B200_ERR_LIMIT;
  // Short calls let the next kernel set up under their tail (us a call, back to back, without and with it: 1003 tokens at stride 16 24.0 and
  // 23.1, 2000 tokens at stride 8 36.7 and 36.0); with more than two units per SM it gains nothing (4096 tokens against 65536 51.9 and
  // 52.2, 32768 tokens 473 and 477).  Dense calls only up to one unit per SM (300 tokens 12.2 and 11.0, 1003 tokens 21.0 and 19.7): beyond
  // that other CTAs get hold of the units left over, and it goes either way (1100 tokens 23.0 and 22.6, 1400 28.3 and 28.9, 1530 31.4 and
  // 31.9, 2000 45.6 and 45.4).  Calls by single tiles gain up to two CTAs per SM, of which the second ones are short (without and with it: 1024
  // tokens 20.4 and 19.4, of 28 heads 19.4 and 18.7, 1180 of 28 heads 23.1 and 22.3), and these have a unit per SM at most.
  p.early_next = units <= (dense ? 1LL : 2LL) * sm_count() ? 1 : 0;
  p.by_units = make_fast_div(causal ? batch * hq : super_rows * (hq / hkv));
  p.by_hq = make_fast_div(hq);
  p.by_batch = make_fast_div(batch);
  p.by_group = make_fast_div(hq / hkv);
  p.by_hkv = make_fast_div(hkv);
  const int32_t* rest = nullptr;
  const int* pair_header = nullptr;
  const int min_share = g_pair_min_share.load();
  if (workspace && !dense && !causal) {
    if (workspace_bytes < order_workspace_bytes(batch, hq, q_len)) return XATTN_B200_ERR_WORKSPACE;
    if ((reinterpret_cast<uintptr_t>(workspace) & 15) != 0) return XATTN_B200_ERR_ARG;
    int32_t* sorted = static_cast<int32_t*>(workspace);
    if ((rc = launch_dependent(attn_order_kernel, dim3(batch * hkv), dim3(kOrderThreads), 0, stream, p, block_cnt, sm_count(), sorted)))
      return rc;
    p.tile_list = sorted;
    p.list_tiles = static_cast<int>(2 * units);
  } else if (workspace && !dense && !out_f32 && pair_path_applies(hq, hkv, k_len)) {
    if ((rc = block_sparse_attn_pair_launch(tmQ, tmK, tmV, p, block_idx, block_cnt, out, workspace, workspace_bytes,
                                            &rest, &pair_header, min_share, status, stream)))
      return rc;
  }
  // (a dependent launch in every case: after the pair kernel, or after whatever kernel produced the block lists)
  const long long sms = sm_count();
  // Two units at a time where the caller knows the lists to be short and there are enough units to go round: at least as many per SM as
  // a list has blocks, so that two of the longest are no more than the tail of the call (32 heads, this kernel: 128K tokens, 111 units
  // per SM, lists of up to 17 blocks, mostly 2: 661 -> 647 us at the power cap and 556 -> 542 in short runs; 9973 tokens, 8 units
  // per SM, 81 -> 84; 58695 tokens, whose few rows of hundreds of blocks then met on one SM, 400 -> 640).  The look at the slots
  // stays out of the other calls: it cost dense ones 1 %.
  const bool two = causal && !dense && !rest && max_list > 0 && units >= 24 * sms && units >= max_list * sms &&
                   static_cast<long long>(batch) * hkv * p.list_k_blocks < 0x7fffffffLL;
  const long long tiles = static_cast<long long>(p.q_blocks) * batch * hq;
  // Causal calls of few tiles give each a CTA of its own, whose streams share its list: up to a tile per SM, dense ones and those with
  // lists of more than 64 key blocks (us, 32 heads, two tiles per CTA and like this; dense, 512 tokens 12.9 and 12.4, against 4096 58 and 38,
  // against 65536 857 and 513; lists of half of the blocks, 512 tokens against 8315 86 and 48, against 65531 580 and 281; of five blocks 24.1
  // and 17.8, 28.0 and 21.9; of two 11.9 in either form.  Shorter rows gain, too: against 2555, 20 blocks, 33.8 and 22.4).
  // With more tiles an SM takes two of them one after the other, which is as many blocks as two at a time, and loads K and V for each: lists
  // go by units of two (1024 tokens against 70000, three blocks, 13.0 and 15.5), and dense calls (1024 against 4096 66 and 71, against 65536
  // 976 and 1184; 900 against 32768 492 and 578), but for two kinds: keys little longer than the queries, where the tiles are of so
  // different lengths that the longest first even the call out (1024 tokens 20.2 and 19.4, 3000 of 12 heads 47.8 and 41.5, against 3750 60.9 and
  // 55.3, 1150 of 28 heads 21.6 and 20.9, 500 of 28 heads in a batch of two 13.3 and 13.2, but against 625 15.6 and 16.3), and more units
  // than SMs, as odd numbers of query blocks make them: the units left over are fetched ahead by CTAs that have one (1150 tokens against
  // 32768 851 and 533, six sequences of 100 against 8192 211 and 150, of which five, 160 tiles, are done in one round, 111 and 150).
  const bool even = 4LL * p.k_len <= 5LL * p.q_len || (units > sms && 4 * tiles > 5 * sms);
  const bool split = causal && !rest && (dense ? tiles <= sms || (tiles <= 2 * sms && even) : tiles <= sms && p.list_k_blocks > 64);
  const unsigned grid = static_cast<unsigned>(rest && units > sms ? sms : (two ? (units + 1) / 2 : (split ? tiles : units)));
  auto launch = [&](auto kern) -> int {
    if (!allow_smem(kern, kAttnSmem))
      return XATTN_B200_ERR_CUDA;
    return launch_dependent(kern, dim3(grid), dim3(kAttnThreads), kAttnSmem, stream, tmQ, tmK,
                            tmV, tmO, p, block_idx, block_cnt, rest, pair_header, min_share, status);
  };
  auto launch_type = [&](auto list, auto pairs, auto parts) -> int {
    constexpr bool kList = decltype(list)::value, kTwo = decltype(pairs)::value, kSplit = decltype(parts)::value;
    return out_f32 ? launch(block_sparse_attn_kernel<true, true, kList, kTwo, kSplit>)
                   : (p.is_bf16 ? launch(block_sparse_attn_kernel<true, false, kList, kTwo, kSplit>) : launch(block_sparse_attn_kernel<false, false, kList, kTwo, kSplit>));
  };
  const auto yes = std::true_type();
  const auto no = std::false_type();
  if (p.tile_list || rest) return launch_type(yes, no, no);
  if (two) return launch_type(no, yes, no);
  return split ? launch_type(no, no, yes) : launch_type(no, no, no);
}

}  // namespace xb
