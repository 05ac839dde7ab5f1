// The threshold selection of one row by one warp (see select.cu for the rule), shared by the selection kernel and by the
// estimate, whose epilogue selects the rows that it has finished.
#pragma once
#include "host_common.cuh"
#include "sm100_primitives.cuh"

namespace xb {

constexpr int kPeelProbe = 8;

// A selection as the callers of the C ABI state it, and as the kernels take it.
struct SelCall {
  const float* attn_sums;
  int batch, heads, q_blocks, k_blocks, bpc, block_offset, causal, diagonal_cleanup;
  double threshold;
  const float* thr_per_head;
  int keep_sink, keep_recent;
  uint8_t* mask;
  int32_t *block_idx, *block_cnt;
  int list_q_blocks, list_k_blocks, list_q_len, list_k_len, band;
  void* rounded;
  int rounded_dtype;
};
struct SelParams {
  int batch, heads, q_blocks, k_blocks;
  int bpc, block_offset, causal, diagonal_cleanup;
  double threshold;
  int keep_sink, keep_recent;
  int list_q_blocks, list_k_blocks, list_q_len, list_k_len;
  int np2;            // k_blocks rounded up to a power of two (>= 32)
  int warps_per_cta;
  int words;          // 32-column words per row
  int vals_bytes, idx_bytes, keys_bytes, per_warp_bytes;   // keys: one sort buffer per CTA, taken in turn by its warps
  int rows_total;
  int vec_in;         // score rows can be read as float4
  int vec_mask;       // mask rows can be written as 16-byte vectors
  int band;           // score rows hold only the chunk's own key blocks [cur, cur + bpc)
  void* rounded;      // (rows in registers) the scores rounded to bf16 / fp16, same layout; null: not wanted
  int rounded_bf16;
  FastDiv by_q_blocks, by_heads, by_bpc;
};

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
// bits of 32-column word t whose column is <= hi
__device__ __forceinline__ uint32_t bits_le(int hi, int t) {
  const int r = hi - 32 * t;
  return r < 0 ? 0u : (r >= 31 ? 0xffffffffu : (2u << r) - 1u);
}

// Post-processing and outputs of one row: `word` is the lane's 32-column word of the taken columns (k_blocks <= 1024).
struct RowOut {
  uint8_t* mask;        // the row of the mask, or null
  int32_t* list;        // the row's list, or null
  int32_t* cnt;
};
__device__ __forceinline__ void finish_row(const SelParams& p, int R, int cur, uint32_t word, int lane, const RowOut& o) {
  const int N = p.k_blocks;
  const uint32_t valid = bits_le(N - 1, lane);
  int hi_keep = N - 1;                             // causal clean-up: columns above are cleared
  if (p.causal) {
    hi_keep = cur + p.bpc - 1;
    if (p.diagonal_cleanup && p.block_offset + R < hi_keep) hi_keep = p.block_offset + R;
  }
  const int recent = p.block_offset + R;
  word &= valid & bits_le(hi_keep, lane);
  if (p.keep_sink && R == 0) word = valid;
  if (p.keep_recent && recent < N && (recent >> 5) == lane) word |= 1u << (recent & 31);
  if (o.mask && 32 * lane < N) {
    uint8_t* mo = o.mask + 32 * lane;
    if (p.vec_mask && 32 * lane + 32 <= N) {
      uint32_t b[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) b[q] = (((word >> (4 * q)) & 15u) * 0x00204081u) & 0x01010101u;
      reinterpret_cast<uint4*>(mo)[0] = make_uint4(b[0], b[1], b[2], b[3]);
      reinterpret_cast<uint4*>(mo)[1] = make_uint4(b[4], b[5], b[6], b[7]);
    } else {
      for (int q = 0; q < 32 && 32 * lane + q < N; ++q) mo[q] = static_cast<uint8_t>((word >> q) & 1u);
    }
  }
  if (o.list) {
    int hi_list = p.list_k_blocks - 1;             // columns the block list may hold
    if (p.causal) {
      // last token of query block R sees keys up to this position (query end aligned to key end)
      int last_q = R * 128 + 127;
      if (last_q > p.list_q_len - 1) last_q = p.list_q_len - 1;
      const int jm = (last_q + (p.list_k_len - p.list_q_len)) >> 7;      // (-1 and less: none)
      if (jm < hi_list) hi_list = jm;
    }
    uint32_t lw = word & bits_le(hi_list, lane);
    int incl = __popc(lw);
    const int own = incl;
#pragma unroll
    for (int s = 1; s < 32; s <<= 1) {
      const int up = __shfl_up_sync(0xffffffffu, incl, s);
      if (lane >= s) incl += up;
    }
    int pos = incl - own;
    while (lw) {
      o.list[pos++] = 32 * lane + __ffs(lw) - 1;
      lw &= lw - 1;
    }
    if (lane == 31) *o.cnt = incl;
  }
}

// Row w of the call by one warp: rows of up to 128 * kVec stored scores and up to 1024 key blocks, in registers; lane l holds
// the columns 128 u + 4 l + e of the stored part (u < kVec, e < 4), zeros past its end.
template <int kVec>
__device__ __forceinline__ void select_values(uint32_t (&v)[4 * kVec], const SelParams& p, const float* thr_per_head, uint8_t* mask_out,
                                              int32_t* idx_out, int32_t* cnt_out, int w, int lane) {
  constexpr unsigned kAll = 0xffffffffu;
  int R, in_chunk, head;
  const int bh = fast_div(w, p.by_q_blocks, R);
  const int N = p.k_blocks;
  const int cur = p.block_offset + fast_div(R, p.by_bpc, in_chunk) * p.bpc;
  const int d = cur + in_chunk;
  const bool f0 = p.causal && cur != 0;            // block 0 forced
  const int n_forced = p.causal ? (f0 ? 2 : 1) : 0;
  const bool lag = n_forced == 1;
  const int n_read = p.band ? p.bpc : N;
  const int col0 = p.band ? cur : 0;
  fast_div(bh, p.by_heads, head);
  const double thr = thr_per_head ? static_cast<double>(ld_written(thr_per_head + head)) : p.threshold;

  // What the estimate returns is the scores in the inputs' type: written here, where the row is in registers anyway (a kernel of
  // its own read the sums once more: estimate and mask of 1003 tokens 25.0 -> 16.8 us, of 8192 49.4 -> 46.6, of 32768 119.2 ->
  // 114.8, of 131072 531 -> 515).
  if (p.rounded) {
    uint16_t* r = static_cast<uint16_t*>(p.rounded) + static_cast<size_t>(w) * n_read;
#pragma unroll
    for (int u = 0; u < kVec; ++u) {
      uint16_t e[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const float f = __uint_as_float(v[4 * u + k]);
        e[k] = p.rounded_bf16 ? __bfloat16_as_ushort(__float2bfloat16_rn(f)) : __half_as_ushort(__float2half_rn(f));
      }
      const int j = u * 128 + 4 * lane;
      if (p.vec_in) {                              // (n_read a multiple of 4: rows of 8-byte vectors)
        if (j < n_read) *reinterpret_cast<uint2*>(r + j) = make_uint2(e[0] | static_cast<uint32_t>(e[1]) << 16, e[2] | static_cast<uint32_t>(e[3]) << 16);
      } else {
#pragma unroll
        for (int k = 0; k < 4; ++k)
          if (j + k < n_read) r[j + k] = e[k];
      }
    }
  }
  // positive floats order like integers; forced and non-positive ones as 0
  double part = 0.0;
  uint32_t at_d = 0u, at_0 = 0u;                   // the forced scores, in the lanes that hold them
  int m = 0;
#pragma unroll
  for (int k = 0; k < 4 * kVec; ++k) {
    const int jj = col0 + (k >> 2) * 128 + 4 * lane + (k & 3);
    const float f = __uint_as_float(v[k]);
    const double df = static_cast<double>(f);
    part += df;
    const bool is_d = p.causal && jj == d, is_0 = f0 && jj == 0;
    if (is_d) at_d = v[k];
    if (is_0) at_0 = v[k];
    if (is_d || is_0 || !(f > 0.f)) v[k] = 0u;
    m += v[k] != 0u;
  }
  const double total = warp_sum(part), fsum = static_cast<double>(__uint_as_float(__reduce_or_sync(kAll, at_d))) +
                                            static_cast<double>(__uint_as_float(__reduce_or_sync(kAll, at_0)));
  const int M = __reduce_add_sync(kAll, m);
  const double req = total * thr;

  uint32_t word = 0u;                              // taken columns, 32 per lane
  auto take = [&](int col) { if (lane == (col >> 5)) word |= 1u << (col & 31); };
  if (p.causal) {
    take(d);
    if (f0) take(0);
  }
  bool untaken = !(req > 0.0);                     // the leading slots of the reference compare 0 < req too
  if (req > 0.0) {
    // Ranks r = 1, 2, ... of the positive scores; prefix[r] = sum of the first r.  K = number of ranks with
    // fsum + prefix[r - 1] < req; without lag the first K ranks are taken, with it the first K + 1.
    int K = 0;
    double above = 0.0;                            // prefix[K]
    bool cut = !(fsum < req);                      // the rank after the first K is refused (without lag)
    // lowest column that holds the bit pattern `best`
    auto column_of = [&](uint32_t best) {
      int c = 0x7fffffff;
#pragma unroll
      for (int k = 4 * kVec - 1; k >= 0; --k)
        if (v[k] == best) c = (k >> 2) * 128 + 4 * lane + (k & 3);
      return __reduce_min_sync(kAll, c);
    };
    auto remove = [&](int c) {                     // (stored column)
#pragma unroll
      for (int k = 0; k < 4 * kVec; ++k)
        if (c == (k >> 2) * 128 + 4 * lane + (k & 3)) v[k] = 0u;
    };
    auto largest = [&]() {
      uint32_t b = 0u;
#pragma unroll
      for (int k = 0; k < 4 * kVec; ++k) b = v[k] > b ? v[k] : b;
      return __reduce_max_sync(kAll, b);
    };
    auto take_next = [&]() {                       // the largest remaining score, lowest column on ties
      const uint32_t b = largest();
      const int c = column_of(b);
      remove(c);
      take(col0 + c);
      return b;
    };
    if (kVec <= 2) {
      // short rows: the first ranks one at a time
#pragma unroll 1
      for (int n = 0; n < kPeelProbe && K < M && !cut; ++n) {
        above += static_cast<double>(__uint_as_float(take_next()));
        ++K;
        cut = !(fsum + above < req);
      }
    }
    if (!cut && K < M) {
      // Bisection for the cut value: scores with pattern > hi are taken (their sum keeps fsum + above below req), the scores
      // in (lo, hi] are undecided.
      uint32_t hi = largest(), lo = 0u;
      int inside = M - K;
#pragma unroll 1
      while (inside > 1 && hi - lo > 1u) {
        const uint32_t mid = lo + ((hi - lo) >> 1);
        double s = 0.0;
        int n = 0;
#pragma unroll
        for (int k = 0; k < 4 * kVec; ++k)
          if (v[k] > mid && v[k] <= hi) {
            s += static_cast<double>(__uint_as_float(v[k]));
            ++n;
          }
        s = warp_sum(s);
        n = __reduce_add_sync(kAll, n);
        if (fsum + (above + s) < req) {
          above += s;
          K += n;
          inside -= n;
          hi = mid;
        } else {
          lo = mid;
          inside = n;
        }
      }
      // the scores in (lo, hi] are equal: in column order until the sum reaches req
      uint32_t tie = 0u;
#pragma unroll
      for (int k = 0; k < 4 * kVec; ++k)
        if (v[k] > lo && v[k] <= hi) tie = v[k];
      tie = __reduce_max_sync(kAll, tie);
      int e = 0;
      const double step = static_cast<double>(__uint_as_float(tie)), base = above;
#pragma unroll 1
      while (e < inside && fsum + above < req) {
        ++e;
        above = base + step * e;
      }
      K += e;
      cut = !(fsum + above < req);
      if (e == inside) {                           // (the usual case: one score, and it is taken)
        hi = lo;
        e = 0;
      }
      // taken so far: every score above hi.  Four ballots hold 128 columns, bit l of ballot e being column 4 l + e; lane
      // 4 u + q builds the word of columns 128 u + 32 q ...
      uint32_t stored = 0u;
#pragma unroll
      for (int u = 0; u < kVec; ++u) {
        uint32_t wd = 0u;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          uint32_t t = (__ballot_sync(kAll, v[4 * u + q] > hi) >> (8 * (lane & 3))) & 0xffu;
          t = (t | (t << 12)) & 0x000f000fu;
          t = (t | (t << 6)) & 0x03030303u;
          t = (t | (t << 3)) & 0x11111111u;
          wd |= t << q;
        }
        if ((lane >> 2) == u) stored = wd;
      }
#pragma unroll
      for (int k = 0; k < 4 * kVec; ++k)
        if (v[k] > hi) v[k] = 0u;
      // from stored columns to key blocks: shifted by col0
      {
        const int t = lane - (col0 >> 5), sh = col0 & 31;
        const uint32_t a = __shfl_sync(kAll, stored, t & 31), b = __shfl_sync(kAll, stored, (t - 1) & 31);
        uint32_t wd = 0u;
        if (t >= 0 && t < 4 * kVec) wd = a << sh;
        if (sh && t >= 1 && t <= 4 * kVec) wd |= b >> (32 - sh);
        word |= wd;
      }
#pragma unroll 1
      for (; e > 0; --e) {                         // some of several equal scores
        const int c = column_of(tie);
        remove(c);
        take(col0 + c);
      }
    }
    int n_taken = K;
    if (lag && K < M) {
      take_next();
      n_taken = K + 1;
    }
    const int n_others = N - n_forced;
    if (n_taken < M) {
      untaken = true;
    } else if (M < n_others) {
      // ranks that hold a zero score (column order): all of them, the first (lag), or none
      const bool first = lag ? K == M : total < req;
      if (!first) {
        untaken = true;
      } else {
        // zero-score columns are the valid ones not taken so far: every positive score is
        const uint32_t zero = ~word & bits_le(N - 1, lane);
        if (total < req) {
          word |= zero;
        } else {
          const int best = __reduce_min_sync(kAll, zero ? 32 * lane + __ffs(zero) - 1 : 0x7fffffff);
          if (best != 0x7fffffff) take(best);
          if (M + 1 < n_others) untaken = true;
        }
      }
    }
  }
  if (untaken) take(0);
  RowOut o;
  o.mask = mask_out ? mask_out + static_cast<size_t>(w) * N : nullptr;
  o.list = nullptr;
  o.cnt = nullptr;
  if (idx_out && cnt_out && R < p.list_q_blocks) {
    const size_t row = static_cast<size_t>(bh) * p.list_q_blocks + R;
    o.list = idx_out + row * p.list_k_blocks;
    o.cnt = cnt_out + row;
  }
  finish_row(p, R, cur, word, lane, o);
}

// The same for a row in memory.
template <int kVec>
__device__ __forceinline__ void select_row(const float* sums, const SelParams& p, const float* thr_per_head, uint8_t* mask_out,
                                           int32_t* idx_out, int32_t* cnt_out, int w, int lane) {
  const int n_read = p.band ? p.bpc : p.k_blocks;
  const float* x = sums + static_cast<size_t>(w) * n_read;
  // The row may be what this warp, or its CTA, has just stored: it is behind a barrier of theirs, and the compiler, which does not know
  // what the loads read, keeps the stores in front of them.
  asm volatile("" ::: "memory");
  // ---- the row, once; scores as bit patterns
  uint32_t v[4 * kVec];
#pragma unroll
  for (int u = 0; u < kVec; ++u) {
    const int j = u * 128 + 4 * lane;
    float4 q = make_float4(0.f, 0.f, 0.f, 0.f);
    if (p.vec_in) {
      const float4 in = ld_written(reinterpret_cast<const float4*>(x + (j < n_read ? j : 0)));      // (no branch per load)
      if (j < n_read) q = in;
    } else {
      if (j < n_read) q.x = ld_written(x + j);
      if (j + 1 < n_read) q.y = ld_written(x + j + 1);
      if (j + 2 < n_read) q.z = ld_written(x + j + 2);
      if (j + 3 < n_read) q.w = ld_written(x + j + 3);
    }
    v[4 * u] = __float_as_uint(q.x); v[4 * u + 1] = __float_as_uint(q.y);
    v[4 * u + 2] = __float_as_uint(q.z); v[4 * u + 3] = __float_as_uint(q.w);
  }
  select_values<kVec>(v, p, thr_per_head, mask_out, idx_out, cnt_out, w, lane);
}

// By a whole CTA, where sums were never finished (a device wait ran out): query blocks [qb0, qb0 + n) of a head select and list
// nothing, so that nobody reads a row of the mask or a list that was never written.
__device__ __forceinline__ void forget_rows(const SelParams& p, uint8_t* mask_out, int32_t* cnt_out, int bh, int qb0, int n) {
  for (int qb = qb0; qb < qb0 + n && qb < p.q_blocks; ++qb) {
    if (mask_out) {
      uint8_t* row = mask_out + (static_cast<size_t>(bh) * p.q_blocks + qb) * p.k_blocks;
      for (int c = threadIdx.x; c < p.k_blocks; c += blockDim.x) row[c] = 0;
    }
    if (cnt_out && threadIdx.x == 0 && qb < p.list_q_blocks) cnt_out[static_cast<size_t>(bh) * p.list_q_blocks + qb] = 0;
  }
}

int select_params(const SelCall& c, SelParams& p);      // checks the call

int select_launch(const SelCall& c, int* status, cudaStream_t stream);

}  // namespace xb
