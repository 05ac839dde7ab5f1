// Definitions shared by the two block-sparse attention kernels (attention.cu: any list length, one work item
// per (head, query block); attention_pair.cu: lists of one or two blocks that the query heads of a kv group share).
#pragma once
#include <math.h>

#include "host_common.cuh"
#include "sm100_primitives.cuh"

namespace xb {

constexpr int kTile16 = 128 * 128 * 2;     // one 128x128 16-bit tile = two 64-column TMA boxes
constexpr int kHalf16 = kTile16 / 2;

struct AttnParams {
  int batch, hq, hkv, q_len, k_len;
  int q_blocks, list_k_blocks;
  int causal, is_bf16;
  float scale_log2;
  int64_t osb, osh, osl;
  FastDiv by_units, by_hq, by_batch, by_group, by_hkv;          // (general kernel: see unit_tile) hq, batch, hq / hkv, hkv
  const int32_t* tile_list;     // general kernel: its tiles, two per unit (null: all, in their natural order)
  int list_tiles;               // entries of that list
  int early_next;               // the kernel after this one may start under the tail
};

__device__ __forceinline__ uint32_t pack16(float lo, float hi, int is_bf16) {
  if (is_bf16) {
    __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&v);
  }
  __half2 v = __floats2half2_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&v);
}

template <bool kBf16> __device__ __forceinline__ uint32_t pack16t(float lo, float hi) { return pack16(lo, hi, kBf16 ? 1 : 0); }

// Development aid, compiled only with -DXB_TRACE: per-role timestamps of the first CTAs, written behind the
// status word (which must then point to a device buffer of at least 64 + 16*14*XB_TRACE_CAP bytes).  Roles: 0/5
// loader, 1/6 MMA issuer of stream 0/1, 4 epilogue, softmax warp (stream s, quad q): q == 0 ? 2 + s : 7 + 3*s + q - 1.
#ifdef XB_TRACE
#ifndef XB_TRACE_CAP
#define XB_TRACE_CAP 4096          // records per role; 14 roles, first CTA only
#endif
__device__ __forceinline__ void xb_trace(int* status, uint32_t& n, int role, uint32_t tag, uint32_t val) {
  if (blockIdx.x >= 1 || !status || n >= XB_TRACE_CAP) return;
  unsigned long long* buf = reinterpret_cast<unsigned long long*>(status) + 8 +
                            2ull * XB_TRACE_CAP * role;
  buf[2 * n] = (static_cast<unsigned long long>(tag) << 32) | val;
  buf[2 * n + 1] = static_cast<unsigned long long>(clock64());
  ++n;
}
#define XB_TRACE_EV(tag, val) xb_trace(status, trace_n, trace_role, (tag), (val))
#else
#define XB_TRACE_EV(tag, val) ((void)0)
#endif

// [128 bytes of columns, rows, column parts, heads, batch] of rows of 128 elements of `elem` bytes (2 or 4): one box
// {128 bytes, `rows`, `parts`, 1, 1} moves `rows` rows of `parts` parts with a single TMA instruction, the parts one after
// the other in shared memory (Q, K, V: both 64-column halves of 16-bit rows).
static inline int make_rows_map(CUtensorMap* m, const void* base, int len, int heads, int batch, int64_t sb, int64_t sh,
                                int64_t sl, uint32_t box_rows, uint32_t box_parts, int elem) {
  const uint64_t cols = 128 / elem;
  const uint64_t dims[5] = {cols, (uint64_t)len, (uint64_t)elem, (uint64_t)heads, (uint64_t)batch};
  // a dimension of extent 1 never moves: give it a harmless valid stride
  const uint64_t s_h = heads > 1 ? (uint64_t)sh * elem : 256, s_b = batch > 1 ? (uint64_t)sb * elem : 256;
  const uint64_t str[4] = {(uint64_t)sl * elem, 128, s_h, s_b};
  const uint32_t box[5] = {(uint32_t)cols, box_rows, box_parts, 1, 1};
  return make_tmap(m, base, elem == 4 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 5, dims, str, box);
}
static inline int make_qkv_map(CUtensorMap* m, const void* base, int len, int heads, int batch, int64_t sb, int64_t sh,
                               int64_t sl, uint32_t box_rows, uint32_t box_halves = 2) {
  return make_rows_map(m, base, len, heads, batch, sb, sh, sl, box_rows, box_halves, 2);
}

// ---------------------------------------------------------------- split between the pair and the general kernel
// Workspace header, in 32-bit words: [0] length of the pair list, [1] length of the list of items left to the
// general kernel, [2..3] / [4..5] 64-bit totals of the blocks listed by all items / by the items on the pair list.
constexpr int kPairRestCount = 1, kPairTotalAll = 2, kPairTotalTaken = 4;
constexpr int kPairMinSharePct = 92;

// The split into two kernels costs a second kernel tail, so nearly all the work has to go to the pair kernel.  (Where the mark
// lies was measured against a general kernel that did not share K/V between two heads; the present one is the faster of the
// two even with 95 % of the blocks on the pair list, 596 against 700 us for the 128K-token layer, so that no call is offered
// the split unless its caller asks for it.)  Both kernels evaluate this after the classify kernel has finished
// and so agree: below the mark (kPairMinSharePct unless the caller set another, see pair_min_share_pct) the pair
// kernel returns at once and the general kernel computes every item.
__device__ __forceinline__ bool pair_path_chosen(const int* header, int min_share_pct) {
  const unsigned long long all = *reinterpret_cast<const volatile unsigned long long*>(header + kPairTotalAll);
  const unsigned long long taken = *reinterpret_cast<const volatile unsigned long long*>(header + kPairTotalTaken);
  return taken * 100ull >= all * static_cast<unsigned long long>(min_share_pct) && taken > 0;
}

}  // namespace xb
