// Decode step: dense attention of ONE query token per sequence against its key cache.
//
// The reference runs it through a third-party single-query kernel (xattn/src/load_llama.py:188-197); the general
// attention kernel here can compute it too, but as a 128-row tile with one valid row per head: a serial walk over the
// cache on as many SMs as there are pairs of heads (128K tokens, 32 / 8 heads: 1.8 ms).
//
// The step reads K and V once and does next to nothing with them, so it is HBM-bound (128K tokens, 8 kv heads: 537 MB, 83 us
// at the measured copy bandwidth; measured 87 us) or, for short caches, pure latency.  Therefore:
//   * the cache is split along its length over the SMs, two CTAs for each or one; a CTA streams its keys through a ring of TMA
//     stages (64 keys of K and V, 32 KiB each): three stages where two CTAs share an SM, up to six where it has one to itself,
//     192 KiB in flight per SM either way, which covers the HBM latency (6.5 TB/s x 1 us / 148 SMs = 44 KiB) several times over;
//   * all query heads of a kv group are rows of one MMA (m16n8k16), so K and V are read once per kv head.  These are warp
//     MMAs on purpose: with at most 16 useful rows a 128-row tcgen05 tile would be seven eighths padding, and the products
//     take under a tenth of the time the bytes do;
//   * every warp takes 16 keys of a stage and keeps a running softmax of its own; the four warps of a CTA are merged
//     through shared memory at the end.  The CTAs of a (batch, kv head) are merged through distributed shared memory where
//     they are a cluster (up to eight: caches of up to 4096 keys, or many heads; sixteen: see decode_splits), and by a small
//     second kernel, launched as a dependent one, where there are more.  The second launch costs the host 2.5 us, which a step
//     on a short cache would pay in full (2011 keys, 8 kv heads: 10.2 us a call with it, 6.0 without), and the second kernel
//     starts when the first has ended; a long cache hides both.
#include <type_traits>

#include "attention_common.cuh"

namespace xb {

constexpr int kDecWarps = 4;
__host__ __device__ constexpr int dec_threads(bool wide) { return kDecWarps * 32 + (wide ? 32 : 0); }   // (wide: and a warp that loads)
constexpr int kDecKeys = 64;                              // keys per stage: 16 per warp
constexpr int kDecTile = kDecKeys * 128 * 2;              // [2 column halves][64 keys][64 columns], 128-byte swizzle
constexpr int kDecStages = 3, kDecMaxStages = 6;          // of the ring: three for two CTAs per SM, up to six for one
constexpr int kDecMaxRows = 16;                           // query heads per kv head
constexpr int dec_smem(int ring) { return ring * 2 * kDecTile + 1024 /*alignment slack*/ + 256 /*barriers*/; }
constexpr float kDecRescale = 8.0f;                       // log2 units: the running maximum moves lazily

struct DecodeParams {
  int batch, hkv, group, k_len, splits, stages;           // stages: 64-key stages of the whole cache
  int cluster;                                            // the splits are a cluster
  int ring;                                               // stages of the ring
  float scale_log2;
  int64_t qsb, qsh, osb, osh;
};

__device__ __forceinline__ void ldsm_x4(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldsm_x4_trans(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
template <bool kBf16>
__device__ __forceinline__ void warp_mma(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  if constexpr (kBf16)
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
  else
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

template <bool kBf16>
__device__ __forceinline__ float2 unpack16t(uint32_t v) {
  if constexpr (kBf16) return __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&v));
  else return __half22float2(*reinterpret_cast<const __half2*>(&v));
}

// part: [batch * hkv][splits][group][128] un-normalised outputs, then [..][splits][group] (max, sum) pairs
// kWide: the kernel for clusters of sixteen, and for smaller ones that have an SM per CTA.  Its ring may be deeper, and it has a warp
// of its own that refills a slot as soon as the four warps are done with it; one of them does it a stage later, which leaves a CTA
// a stage less in flight (30000 keys, 4 kv heads: 17.8 us a call against 26.3, before the second term below).  The others, two CTAs
// per SM, have enough in flight, and with that warp their merge kernel came 5 us later.
// kSixteen: clusters of sixteen, up to eight otherwise.  Each part of the cache has a maximum of its own, whose exponential is exact, so
// that these parts, fewer than those of two CTAs per SM, would round a little more: they multiply the probabilities in two 16-bit
// terms.  Clusters of up to eight have the same parts in either kernel, and one term in both: a sequence's result does not depend on
// the batch that it is in.
template <bool kBf16, bool kWide, bool kSixteen>
__global__ void __launch_bounds__(dec_threads(kWide), 2)
decode_attn_kernel(const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV,
                   const uint16_t* __restrict__ q, const DecodeParams p, float* __restrict__ part,
                   float2* __restrict__ part_ml, uint16_t* __restrict__ out, int* status) {
  const int ring = kWide ? p.ring : kDecStages;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + ring * 2 * kDecTile);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(bars + 2 * kDecMaxStages);
  const uint32_t full0 = smem_u32(bars), empty0 = smem_u32(bars + kDecMaxStages);
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int split = blockIdx.x, g = blockIdx.y, b = blockIdx.z;
  // stages [s0, s1) of the cache
  const int s0 = static_cast<int>(static_cast<long long>(p.stages) * split / p.splits);
  const int s1 = static_cast<int>(static_cast<long long>(p.stages) * (split + 1) / p.splits);
  if (threadIdx.x == 0) {
    for (int s = 0; s < ring; ++s) {
      mbar_init(full0 + 8 * s, 1);
      mbar_init(empty0 + 8 * s, kDecWarps);
    }
    *abort_flag = 0;
    fence_mbar_init();
  }
  __syncthreads();
  pdl_launch_dependents();              // the next kernel may take its place; it waits for this grid to end
  pdl_wait();
  auto load_stage = [&](int i, int st) {        // one thread: the CTA's i-th stage, into slot st
    const uint32_t dst = smem_u32(smem) + st * 2 * kDecTile;
    mbar_expect_tx(full0 + 8 * st, 2 * kDecTile);
    tma_load_5d(dst, &tmK, full0 + 8 * st, 0, (s0 + i) * kDecKeys, 0, g, b);
    tma_load_5d(dst + kDecTile, &tmV, full0 + 8 * st, 0, (s0 + i) * kDecKeys, 0, g, b);
  };
  const int n = s1 - s0;
  constexpr int kDecThreads = dec_threads(kWide);
  if (!kWide && threadIdx.x == 0)
    for (int i = 0; i < ring && i < n; ++i) load_stage(i, i);
  float o[16][4];
  float m[2], l[2];                                        // rows lane / 4 and lane / 4 + 8
  int st = 0, last = ring - 1;                             // this stage's slot (of the loading warp: to load), the slot of the one before
  uint32_t ph = kWide && warp == kDecWarps ? 1 : 0, last_ph = 1;       // and the phases of their barriers
  int loads = 0;
  auto pass = [&](auto two_terms) {                        // the CTA's part of the cache, with the probabilities in one or two terms
    constexpr bool kTwo = decltype(two_terms)::value;
    if (kWide && warp == kDecWarps) {
      if (lane == 0) {
        for (int i = 0; i < n; ++i, ++loads) {
          if (loads >= ring && !mbar_wait(empty0 + 8 * st, ph, abort_flag)) break;
          load_stage(i, st);
          if (++st == ring) { st = 0; ph ^= 1; }
        }
      }
      __syncwarp();
    }
    if (warp < kDecWarps) {
      // Q as A operand: rows = query heads of the group (rows past it zero), 8 steps of 16 columns
      uint32_t qa[8][4];
      {
        const int r0 = lane >> 2, c0 = (lane & 3) * 2;
        const uint16_t* qg = q + b * p.qsb + static_cast<int64_t>(g) * p.group * p.qsh;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int r = r0 + 8 * h;
#pragma unroll
          for (int k = 0; k < 8; ++k) qa[k][h] = qa[k][2 + h] = 0u;
          if (r < p.group) {
            const uint16_t* row = qg + r * p.qsh + c0;
#pragma unroll
            for (int k = 0; k < 8; ++k)
#pragma unroll
              for (int e = 0; e < 2; ++e) qa[k][2 * e + h] = ld_written(reinterpret_cast<const uint32_t*>(row + 16 * k + 8 * e));
          }
        }
      }
#pragma unroll
      for (int t = 0; t < 16; ++t)
#pragma unroll
        for (int e = 0; e < 4; ++e) o[t][e] = 0.f;
      m[0] = m[1] = -INFINITY;
      l[0] = l[1] = 0.f;
      // ldmatrix addresses: lane's row inside the warp's 16 keys; chunk c of 16 bytes of row r sits at chunk c ^ (r & 7)
      const int krow = warp * 16 + (lane & 7) + ((lane >> 4) << 3), kchunk = (lane >> 3) & 1;   // K: keys 0-7 | 8-15, columns 0-7 | 8-15
      const int vrow = warp * 16 + (lane & 7) + (((lane >> 3) & 1) << 3), vchunk = lane >> 4;   // V: the same, transposed on load
      bool ok = true;
      for (int i = 0; i < n; ++i) {
        if (!__all_sync(0xffffffffu, mbar_wait(full0 + 8 * st, ph, abort_flag))) break;
        const uint32_t kt = smem_u32(smem) + st * 2 * kDecTile, vt = kt + kDecTile;
        float s[2][4] = {};                                    // keys 0-7, 8-15 of the warp
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          uint32_t kb[4];
          ldsm_x4(kt + (k >> 2) * (kDecTile / 2) + krow * 128 + (((((k & 3) << 1) | kchunk) ^ (krow & 7)) << 4), kb);
          warp_mma<kBf16>(s[0], qa[k], kb[0], kb[1]);
          warp_mma<kBf16>(s[1], qa[k], kb[2], kb[3]);
        }
        const int key0 = (s0 + i) * kDecKeys + warp * 16 + (lane & 3) * 2;
        if ((s0 + i + 1) * kDecKeys > p.k_len) {
#pragma unroll
          for (int t = 0; t < 2; ++t)
#pragma unroll
            for (int e = 0; e < 4; ++e)
              if (key0 + 8 * t + (e & 1) >= p.k_len) s[t][e] = -INFINITY;
        }
        float mx[2];
        bool grow = false;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          mx[h] = fmaxf(fmaxf(s[0][2 * h], s[0][2 * h + 1]), fmaxf(s[1][2 * h], s[1][2 * h + 1]));
          mx[h] = fmaxf(mx[h], __shfl_xor_sync(0xffffffffu, mx[h], 1));
          mx[h] = fmaxf(mx[h], __shfl_xor_sync(0xffffffffu, mx[h], 2)) * p.scale_log2;
          grow |= mx[h] > m[h] + kDecRescale;                  // (-inf + 8 is -inf: the first finite maximum counts)
        }
        if (__any_sync(0xffffffffu, grow)) {
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const float mn = fmaxf(m[h], mx[h]);
            const float alpha = m[h] == -INFINITY ? 0.f : fast_exp2(m[h] - mn);
            m[h] = mn;
            l[h] *= alpha;
#pragma unroll
            for (int t = 0; t < 16; ++t) {
              o[t][2 * h] *= alpha;
              o[t][2 * h + 1] *= alpha;
            }
          }
        }
        uint32_t pa[4], pl[4];                                 // (kTwo) pl: what the rounding of pa leaves
#pragma unroll
        for (int t = 0; t < 2; ++t)
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const float mr = m[h] == -INFINITY ? 0.f : m[h];
            const float p0 = fast_exp2(fmaf(s[t][2 * h], p.scale_log2, -mr)), p1 = fast_exp2(fmaf(s[t][2 * h + 1], p.scale_log2, -mr));
            l[h] += p0 + p1;
            pa[2 * t + h] = pack16t<kBf16>(p0, p1);
            if constexpr (kTwo) {
              const float2 r = unpack16t<kBf16>(pa[2 * t + h]);
              pl[2 * t + h] = pack16t<kBf16>(p0 - r.x, p1 - r.y);
            }
          }
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          uint32_t vb[4];
          ldsm_x4_trans(vt + (c >> 2) * (kDecTile / 2) + vrow * 128 + (((((c & 3) << 1) | vchunk) ^ (vrow & 7)) << 4), vb);
          warp_mma<kBf16>(o[2 * c], pa, vb[0], vb[1]);
          warp_mma<kBf16>(o[2 * c + 1], pa, vb[2], vb[3]);
          if constexpr (kTwo) {
            warp_mma<kBf16>(o[2 * c], pl, vb[0], vb[1]);
            warp_mma<kBf16>(o[2 * c + 1], pl, vb[2], vb[3]);
          }
        }
        if (i + ring < n) fence_proxy_async_smem();      // every lane's reads of the stage come before the TMA writes that refill it
        __syncwarp();
        if (lane == 0) mbar_arrive(empty0 + 8 * st);
        if constexpr (!kWide) {
          if (threadIdx.x == 0 && i > 0 && i - 1 + ring < n) {
            // the stage before this one is refilled: by now every warp is done with it, or nearly
            if (mbar_wait(empty0 + 8 * last, last_ph, abort_flag)) load_stage(i - 1 + ring, last);
            else ok = false;
          }
          ok = __shfl_sync(0xffffffffu, ok, 0);
          if (!ok) break;
          last = st;
          last_ph = ph;
        }
        if (++st == ring) { st = 0; ph ^= 1; }
      }
      // row sums over the four lanes of a row
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        l[h] += __shfl_xor_sync(0xffffffffu, l[h], 1);
        l[h] += __shfl_xor_sync(0xffffffffu, l[h], 2);
      }
    }
  };
  pass(std::integral_constant<bool, kSixteen>());
  // every stage has been read: the ring becomes the exchange buffer
  if constexpr (kSixteen) {
    // The products of an infinite value with the second terms, zero or of either sign, are NaN: where a result is not finite the cache is
    // read again for the first terms alone.  (As a copy of the pass: a choice inside it made every call longer, 30000 keys, 4 kv heads,
    // 20.2 -> 26.0 us around the products of a step, 23.4 around all of them.)
    float check = 0.f;
    if (warp < kDecWarps) {
#pragma unroll
      for (int t = 0; t < 16; ++t)
#pragma unroll
        for (int e = 0; e < 4; ++e) check = fmaf(o[t][e], 0.f, check);
    }
    if (__syncthreads_or(check != 0.f) && !*abort_flag) {
      fence_proxy_async_smem();                            // (the reads of the last stages come before the TMA writes that follow)
      __syncthreads();
      pass(std::false_type());
      __syncthreads();
    }
  } else {
    __syncthreads();
  }
  const bool aborted = *abort_flag != 0;
  if (aborted) {
    const long long t0 = clock64();
    while (clock64() - t0 < 2000000) { __nanosleep(1000); }      // let copies in flight land
    if (threadIdx.x == 0 && status) atomicExch(status, static_cast<int>(kDevWaitTimeout));
    __syncthreads();
  }
  float* xo = reinterpret_cast<float*>(smem);                                    // [warp][16 rows][128]
  float2* xml = reinterpret_cast<float2*>(smem + kDecWarps * kDecMaxRows * 128 * 4);     // [warp][16 rows]
  float* res = xo + kDecWarps * kDecMaxRows * 128 + 2 * kDecWarps * kDecMaxRows;          // [16 rows][128], the CTA's part
  float2* res_ml = reinterpret_cast<float2*>(res + kDecMaxRows * 128);                    // [16 rows]
  if (warp < kDecWarps) {
    const int r0 = lane >> 2, c0 = (lane & 3) * 2;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int r = r0 + 8 * h;
      if (r < p.group) {
#pragma unroll
        for (int t = 0; t < 16; ++t)
          *reinterpret_cast<float2*>(xo + (warp * kDecMaxRows + r) * 128 + t * 8 + c0) = make_float2(o[t][2 * h], o[t][2 * h + 1]);
        if ((lane & 3) == 0) xml[warp * kDecMaxRows + r] = make_float2(m[h], l[h]);
      }
    }
  }
  __syncthreads();
  for (int e = threadIdx.x; e < p.group * 64; e += kDecThreads) {                // two columns of a row
    const int r = e >> 6, c = (e & 63) * 2;
    float mm = -INFINITY;
#pragma unroll
    for (int w = 0; w < kDecWarps; ++w) mm = fmaxf(mm, xml[w * kDecMaxRows + r].x);
    float a0 = 0.f, a1 = 0.f, ll = 0.f;
#pragma unroll
    for (int w = 0; w < kDecWarps; ++w) {
      const float2 ml = xml[w * kDecMaxRows + r];
      const float f = ml.x == -INFINITY ? 0.f : fast_exp2(ml.x - mm);
      const float2 v = *reinterpret_cast<const float2*>(xo + (w * kDecMaxRows + r) * 128 + c);
      a0 += v.x * f;
      a1 += v.y * f;
      ll += ml.y * f;
    }
    if (p.splits == 1) {
      const float inv = ll > 0.f ? 1.f / ll : 0.f;
      *reinterpret_cast<uint32_t*>(out + b * p.osb + static_cast<int64_t>(g * p.group + r) * p.osh + c) =
          pack16t<kBf16>(a0 * inv, a1 * inv);
    } else if (p.cluster) {
      *reinterpret_cast<float2*>(res + r * 128 + c) = make_float2(a0, a1);
      if (c == 0) res_ml[r] = make_float2(mm, ll);
    } else {
      const size_t row = (static_cast<size_t>(b * p.hkv + g) * p.splits + split) * p.group + r;
      *reinterpret_cast<float2*>(part + row * 128 + c) = make_float2(a0, a1);
      if (c == 0) part_ml[row] = make_float2(mm, ll);
    }
  }
  if (p.cluster) {
    // every CTA merges its share of the outputs, two columns of a row at a time
    cluster_sync_all();
    for (int e = split * kDecThreads + threadIdx.x; e < p.group * 64; e += p.splits * kDecThreads) {
      const int r = e >> 6, c = (e & 63) * 2;
      float a0 = 0.f, a1 = 0.f, ll = 0.f;
      auto merge = [&](auto most) {                        // parts of up to `most` CTAs
        constexpr int kParts = decltype(most)::value;
        float2 ml[kParts], v[kParts];
        float mm = -INFINITY;
#pragma unroll
        for (int s = 0; s < kParts; ++s) {
          ml[s] = make_float2(-INFINITY, 0.f);
          v[s] = make_float2(0.f, 0.f);
          if (s < p.splits) {
            ml[s] = ld_shared_cluster_f2(mapa_shared(smem_u32(res_ml + r), s));
            v[s] = ld_shared_cluster_f2(mapa_shared(smem_u32(res + r * 128 + c), s));
          }
          mm = fmaxf(mm, ml[s].x);
        }
#pragma unroll
        for (int s = 0; s < kParts; ++s) {
          const float f = ml[s].x == -INFINITY ? 0.f : fast_exp2(ml[s].x - mm);
          a0 += v[s].x * f;
          a1 += v[s].y * f;
          ll += ml[s].y * f;
        }
      };
      merge(std::integral_constant<int, kSixteen ? 16 : 8>());
      const float inv = ll > 0.f ? 1.f / ll : 0.f;
      *reinterpret_cast<uint32_t*>(out + b * p.osb + static_cast<int64_t>(g * p.group + r) * p.osh + c) =
          pack16t<kBf16>(a0 * inv, a1 * inv);
    }
    cluster_sync_all();                  // nobody leaves while its part may still be read
  }
}

// One CTA per (batch, query head), a thread per column: the splits' parts into the output.
template <bool kBf16>
__global__ void __launch_bounds__(128)
decode_merge_kernel(const DecodeParams p, const float* __restrict__ part, const float2* __restrict__ part_ml,
                    uint16_t* __restrict__ out) {
  pdl_launch_dependents();
  pdl_wait();
  const int hq = p.hkv * p.group;
  const int b = blockIdx.x / hq, h = blockIdx.x - b * hq;
  const int g = h / p.group, r = h - g * p.group;
  const size_t row0 = static_cast<size_t>(b * p.hkv + g) * p.splits * p.group + r;
  constexpr int kAhead = 8;               // loads in flight: a split's part waits for its factor otherwise (128K tokens: 90 us)
  float mm = -INFINITY;
#pragma unroll 1
  for (int s0 = 0; s0 < p.splits; s0 += kAhead) {
    float2 ml[kAhead];
#pragma unroll
    for (int j = 0; j < kAhead; ++j)
      ml[j] = s0 + j < p.splits ? ld_written(part_ml + row0 + static_cast<size_t>(s0 + j) * p.group) : make_float2(-INFINITY, 0.f);
#pragma unroll
    for (int j = 0; j < kAhead; ++j) mm = fmaxf(mm, ml[j].x);
  }
  float a = 0.f, ll = 0.f;
#pragma unroll 1
  for (int s0 = 0; s0 < p.splits; s0 += kAhead) {
    float2 ml[kAhead];
    float x[kAhead];
#pragma unroll
    for (int j = 0; j < kAhead; ++j) {
      const size_t row = row0 + static_cast<size_t>(s0 + j) * p.group;
      ml[j] = s0 + j < p.splits ? ld_written(part_ml + row) : make_float2(-INFINITY, 0.f);
      x[j] = s0 + j < p.splits ? ld_written(part + row * 128 + threadIdx.x) : 0.f;
    }
#pragma unroll
    for (int j = 0; j < kAhead; ++j) {
      const float f = ml[j].x == -INFINITY ? 0.f : fast_exp2(ml[j].x - mm);
      a += x[j] * f;
      ll += ml[j].y * f;
    }
  }
  const float v = ll > 0.f ? a / ll : 0.f;
  uint16_t* o = out + b * p.osb + h * p.osh + threadIdx.x;
  *o = static_cast<uint16_t>(pack16t<kBf16>(v, 0.f));
}

// Number of splits: two CTAs per SM over all (batch, kv head) pairs, at least two stages each (a split costs a CTA's start
// and its row of the merge, about what two stages take).  Up to eight of them are a cluster, whose size is a power of two;
// so are those of caches of up to 4096 keys, where eight CTAs of eight stages take about as long as the second kernel.
// Longer caches: clusters of sixteen, where all of them fit on the chip at the same time (14 on this one with two CTAs per SM, seven
// with one), rather than more CTAs and a second kernel, which starts when the first has ended and reads what it wrote.  us a
// call, 1 sequence, 32 / 8 heads: 4200 keys 12.5 -> 8.3, 12717 18.8 -> 15.4, 30000 29.1 -> 27.8; 28 / 4 heads: 30000 27.4 -> 20.5, 60000
// 36.6 -> 35.2; 8 / 1 heads, 30000 keys: 45 -> 19.  Up to 128 of 148 SMs stream then, and the time per key is a
// third longer than with all of them (rings of three) or grows with the CTA's own share (deep rings, fewer heads): from about 40 and
// 66 stages per CTA on the second kernel is the lesser cost.
constexpr int kDecClusterMax = 8, kDecClusterStages = 64, kDecClusterWide = 16;
constexpr int kDecWideStages = 36, kDecWideStagesDeep = 64;      // stages per CTA up to which sixteen are the faster way (rings of 3, of 6)
static int wide_clusters(bool deep);                     // clusters of sixteen, with rings of three or six, that fit on the device at a time
static int decode_splits(int batch, int hkv, int k_len, int& cluster) {
  const int stages = (k_len + kDecKeys - 1) / kDecKeys;
  const long long heads = static_cast<long long>(batch) * hkv;
  long long s = 2LL * sm_count() / heads;
  if (s > stages / 2) s = stages / 2;
  if (s > kDecClusterMax && (stages <= kDecClusterStages || s < kDecClusterMax * 3 / 2)) s = kDecClusterMax;
  const bool sixteen = s >= kDecClusterWide && heads <= wide_clusters(false) &&
                       stages <= kDecClusterWide * (heads <= wide_clusters(true) ? kDecWideStagesDeep : kDecWideStages);
  if (sixteen) s = kDecClusterWide;
  cluster = s > 1 && (s <= kDecClusterMax || sixteen) ? 1 : 0;         // (sixteen splits that come out as such are not one)
  if (cluster)
    while (s & (s - 1)) s &= s - 1;
  return s < 1 ? 1 : static_cast<int>(s);
}

size_t decode_workspace_bytes(int batch, int hq, int hkv, int k_len) {
  if (batch < 1 || hq < 1 || hkv < 1 || hq % hkv != 0 || hq / hkv > kDecMaxRows || k_len < 1) return 0;
  int cluster = 0;
  const int splits = decode_splits(batch, hkv, k_len, cluster);
  if (cluster || splits == 1) return 0;
  return static_cast<size_t>(batch) * hq * splits * (128 * sizeof(float) + sizeof(float2));
}

// once per kernel and device: its shared memory, and (wide) clusters of sixteen
template <typename K>
static bool dec_allow(K kern, bool wide) {
  return once_per_device(reinterpret_cast<const void*>(kern), [&]() {
    const bool ok = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, dec_smem(kDecMaxStages)) == cudaSuccess &&
                    (!wide || cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess);
    if (!ok) cudaGetLastError();
    return ok ? 1 : 0;
  }) > 0;
}
static int wide_clusters(bool deep) {
  static const char keys[2] = {};
  return once_per_device(&keys[deep], [&]() {
    const auto kern = decode_attn_kernel<true, true, true>;
    if (!dec_allow(kern, true)) return 0;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(kDecClusterWide, 64, 1);
    cfg.blockDim = dim3(dec_threads(true), 1, 1);
    cfg.dynamicSmemBytes = dec_smem(deep ? kDecMaxStages : kDecStages);
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = kDecClusterWide;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int m = 0;
    if (cudaOccupancyMaxActiveClusters(&m, kern, &cfg) != cudaSuccess) {
      cudaGetLastError();
      return 0;
    }
    return m;
  });
}

int decode_launch(const void* q, const void* k, const void* v, int dtype, int batch, int hq, int hkv, int k_len,
                  int head_dim, int64_t qsb, int64_t qsh, int64_t ksb, int64_t ksh, int64_t ksl, int64_t vsb, int64_t vsh,
                  int64_t vsl, float scale, void* out, int64_t osb, int64_t osh, void* workspace, size_t workspace_bytes,
                  int* status, cudaStream_t stream) {
  if (!q || !k || !v || !out) return XATTN_B200_ERR_ARG;
  if (dtype != XATTN_B200_BF16 && dtype != XATTN_B200_F16) return XATTN_B200_ERR_ARG;
  if (head_dim != 128 || batch < 1 || hq < 1 || hkv < 1 || hq % hkv != 0 || k_len < 1 || !(scale > 0.f)) return XATTN_B200_ERR_ARG;
  // a dimension of extent 1 never moves: its stride is no matter
  if (batch == 1) qsb = osb = 0;
  if (hq == 1) qsh = osh = 0;
  if (((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(out)) & 3) || ((qsb | qsh | osb | osh) & 1)) return XATTN_B200_ERR_ARG;
  if (hq / hkv > kDecMaxRows || hkv > 65535 || batch > 65535) return XATTN_B200_ERR_LIMIT;
  int rc;
  if ((rc = check_sm100())) return rc;
  DecodeParams p;
  p.batch = batch; p.hkv = hkv; p.group = hq / hkv; p.k_len = k_len;
  p.stages = (k_len + kDecKeys - 1) / kDecKeys;
  p.splits = decode_splits(batch, hkv, k_len, p.cluster);
  // where every CTA has an SM to itself its ring is deeper
  p.ring = kDecStages;
  const long long heads = static_cast<long long>(batch) * hkv;
  if (p.splits > kDecClusterMax ? p.cluster && heads <= wide_clusters(true) : 4 * p.splits * heads <= 3LL * sm_count()) {
    const int most = (p.stages + p.splits - 1) / p.splits;
    p.ring = most < kDecStages ? kDecStages : (most > kDecMaxStages ? kDecMaxStages : most);
  }
  p.scale_log2 = scale * 1.4426950408889634f;
  p.qsb = qsb; p.qsh = qsh; p.osb = osb; p.osh = osh;
  const size_t need = decode_workspace_bytes(batch, hq, hkv, k_len);
  if (need && (!workspace || workspace_bytes < need)) return XATTN_B200_ERR_WORKSPACE;
  if (reinterpret_cast<uintptr_t>(workspace) & 15) return XATTN_B200_ERR_ARG;
  float* part = static_cast<float*>(workspace);
  float2* part_ml = reinterpret_cast<float2*>(part + static_cast<size_t>(batch) * hq * p.splits * 128);
  CUtensorMap tmK, tmV;
  if ((rc = make_qkv_map(&tmK, k, k_len, hkv, batch, ksb, ksh, ksl, kDecKeys))) return rc;
  if ((rc = make_qkv_map(&tmV, v, k_len, hkv, batch, vsb, vsh, vsl, kDecKeys))) return rc;
  const bool wide = p.cluster && (p.splits > kDecClusterMax || p.ring > kDecStages);
  auto launch = [&](auto kern, auto merge) -> int {
    if (!dec_allow(kern, wide))
      return XATTN_B200_ERR_CUDA;
    const int r = launch_dependent_clusters(kern, p.cluster ? p.splits : 1, dim3(p.splits, hkv, batch), dim3(dec_threads(wide)), dec_smem(p.ring), stream,
                                            tmK, tmV, static_cast<const uint16_t*>(q), p, part, part_ml, static_cast<uint16_t*>(out), status);
    if (r || p.cluster || p.splits == 1) return r;
    return launch_dependent(merge, dim3(batch * hq), dim3(128), 0, stream, p, static_cast<const float*>(part),
                            static_cast<const float2*>(part_ml), static_cast<uint16_t*>(out));
  };
  auto launch_type = [&](auto bf16) -> int {
    constexpr bool kBf16 = decltype(bf16)::value;
    if (!wide) return launch(decode_attn_kernel<kBf16, false, false>, decode_merge_kernel<kBf16>);
    return p.splits > kDecClusterMax ? launch(decode_attn_kernel<kBf16, true, true>, decode_merge_kernel<kBf16>)
                                     : launch(decode_attn_kernel<kBf16, true, false>, decode_merge_kernel<kBf16>);
  };
  return dtype == XATTN_B200_BF16 ? launch_type(std::true_type()) : launch_type(std::false_type());
}

}  // namespace xb
