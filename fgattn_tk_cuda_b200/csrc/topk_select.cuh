// Top-k key selection per query block (the alternative list producer of the reference,
// qk_topkmask_indices in python/spattn/mask_utils.py:389-417): score(query block, key) =
// mean of the block's query rows . key * scale; the select_k keys with the largest score become
// the block's list, in descending score order.
//
// Three kernels:
//   qblock_mean_kernel   : block means of q in fp32, written as a bf16 pair hi + lo (hi = bf16(mean),
//                          lo = bf16(mean - hi)), so that two bf16 tensor-core products reproduce
//                          the fp32 mean to ~2^-17 relative.  HBM-bound read of q.
//   topk_scores_kernel   : scores = (hi + lo) . k^T on tcgen05 (tiles of 128 query blocks x 128 keys,
//                          accumulators in TMEM), written as fp32 rows; columns past kv_len hold -inf.
//   topk_select_kernel   : per row a threshold from a sample and one sweep that collects, or an interval-narrowing
//                          histogram select (2048 bins per sweep) for the k-th largest score, ordered tie
//                          handling (smallest key index first), then the selected (score, index) pairs put in
//                          order in shared memory, or their bits set.
#pragma once
#include "sm100_ptx.cuh"

namespace fg {

// grid (n_blocks, BH), 256 threads.
template <int D>
__global__ void __launch_bounds__(256)
qblock_mean_kernel(const __nv_bfloat16* q, __nv_bfloat16* qm_hi,
                   __nv_bfloat16* qm_lo, int S, int n_blocks, int blocksz, float scale) {
  constexpr int kChunks = D / 8;                 // 16-byte chunks per row
  constexpr int kGroups = 256 / kChunks;         // row groups working in parallel
  __shared__ float part[kGroups][D];
  const int blk = blockIdx.x, bh = blockIdx.y, tid = threadIdx.x;
  grid_trigger();
  grid_wait();
  const int chunk = tid % kChunks, grp = tid / kChunks;
  const int r0 = blk * blocksz, rows = min(blocksz, S - r0);
  float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  const __nv_bfloat16* base = q + (size_t(bh) * S + r0) * D + chunk * 8;
  for (int r = grp; r < rows; r += kGroups) {
    const uint4 v = *reinterpret_cast<const uint4*>(base + size_t(r) * D);
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      acc[2 * i] += __uint_as_float(w[i] << 16);
      acc[2 * i + 1] += __uint_as_float(w[i] & 0xffff0000u);
    }
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) part[grp][chunk * 8 + i] = acc[i];
  __syncthreads();
  if (tid < D) {
    float s = 0.f;
#pragma unroll 8
    for (int g = 0; g < kGroups; ++g) s += part[g][tid];
    const float mean = s / float(rows) * scale;
    const __nv_bfloat16 hi = __float2bfloat16_rn(mean);
    const size_t off = (size_t(bh) * n_blocks + blk) * D + tid;
    qm_hi[off] = hi;
    qm_lo[off] = __float2bfloat16_rn(mean - __bfloat162float(hi));
  }
}

struct TopkScoreParams {
  float* scores;       // [BH, n_blocks, s_stride]
  int* err;
  int n_blocks, kv_len, s_stride;
  int k_tiles, q_tiles, n_tiles;       // 128-key tiles of a unit, 128-query-block tiles of a unit, score tiles in all
};

template <int D>
struct TopkScoreCfg {
  static constexpr int kHalves = D / 64;
  static constexpr int kTileBytes = 128 * D * 2;
  static constexpr int kStages = 4;
  static constexpr int kOffK = 2 * kTileBytes;                        // behind the block means, hi and lo
  static constexpr int kOffBar = kOffK + kStages * kTileBytes;
  static constexpr int kSmemBytes = kOffBar + 256 + 1024;
  static constexpr int kWarpProd = 8, kWarpIss = 9;
  static constexpr int kThreads = 32 * 10;
};

enum : int { TS_Q_FULL = 0, TS_Q_EMPTY = 1, TS_K_FULL = 2, TS_K_EMPTY = 6, TS_S_FULL = 10, TS_S_EMPTY = 12, TS_COUNT = 14 };

// Score tiles (128 query blocks x 128 keys), key tiles of one query tile in a row, are cut into as many contiguous shares as
// there are thread blocks (one per SM): the means are loaded once per share and unit, K streams through a ring, the
// products go to two accumulators in turn, and a warpgroup each takes them from there to memory, a row per thread in
// 32-byte pieces, which are whole sectors.  What is left is the writing of the scores.  12 heads, 256 query blocks x 32760
// keys, D = 128 (402 MB): 0.113 ms; 0.146 with a thread block per tile and rows put together in shared memory.
// Warps 0-3 / 4-7: even / odd tiles of the share, warp 8 TMA producer, warp 9 UMMA issuer.
template <int D>
__global__ void __launch_bounds__(TopkScoreCfg<D>::kThreads, 1)
topk_scores_kernel(const __grid_constant__ CUtensorMap m_hi, const __grid_constant__ CUtensorMap m_lo,
                   const __grid_constant__ CUtensorMap mk, const TopkScoreParams p) {
  using Cfg = TopkScoreCfg<D>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const uint32_t sbase = smem_u32(smem);
  auto bar = [&](int i) -> uint32_t { return sbase + Cfg::kOffBar + 8u * uint32_t(i); };
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + Cfg::kOffBar + 8 * TS_COUNT);
  AbortState* ab = reinterpret_cast<AbortState*>(smem + Cfg::kOffBar + 8 * TS_COUNT + 8);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int from = int((long long)p.n_tiles * blockIdx.x / gridDim.x), to = int((long long)p.n_tiles * (blockIdx.x + 1) / gridDim.x);

  if (tid == 0) {
    ab->flag = 0;
    mbar_init(bar(TS_Q_FULL), 1);
    mbar_init(bar(TS_Q_EMPTY), 1);
    for (int i = 0; i < Cfg::kStages; ++i) {
      mbar_init(bar(TS_K_FULL + i), 1);
      mbar_init(bar(TS_K_EMPTY + i), 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(bar(TS_S_FULL + i), 1);
      mbar_init(bar(TS_S_EMPTY + i), 128);
    }
    mbar_fence_init();
  }
  grid_trigger();
  grid_wait();                         // for the means; before tensor memory is taken (launch_behind)
  if (warp == Cfg::kWarpProd) {
    __syncwarp();
    tmem_alloc(smem_u32(tmem_slot), 256);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  if (warp == Cfg::kWarpProd) {
    if (lane == 0) {
      tma_prefetch_desc(&m_hi);
      tma_prefetch_desc(&m_lo);
      tma_prefetch_desc(&mk);
      bool ok = true;
      int n_q = 0, g = 0;                                  // query tiles and K tiles requested so far
      for (int i = from; i < to; ++i, ++g) {
        const int row = i / p.k_tiles, unit = row / p.q_tiles;          // (unit, query tile)
        if (i == from || i % p.k_tiles == 0) {
          if (n_q > 0) ok = mbar_wait_relaxed(bar(TS_Q_EMPTY), (n_q - 1) & 1, ab, p.err, 3103);
          if (!ok) break;
          mbar_arrive_expect_tx(bar(TS_Q_FULL), 2 * Cfg::kTileBytes);
          for (int h = 0; h < Cfg::kHalves; ++h) {
            tma_load_3d(sbase + h * 16384, &m_hi, bar(TS_Q_FULL), h * 64, (row - unit * p.q_tiles) * 128, unit);
            tma_load_3d(sbase + Cfg::kTileBytes + h * 16384, &m_lo, bar(TS_Q_FULL), h * 64, (row - unit * p.q_tiles) * 128, unit);
          }
          ++n_q;
        }
        const int st = g % Cfg::kStages, f = g / Cfg::kStages;
        if (f > 0) ok = mbar_wait_relaxed(bar(TS_K_EMPTY + st), (f - 1) & 1, ab, p.err, 3104);
        if (!ok) break;
        mbar_arrive_expect_tx(bar(TS_K_FULL + st), Cfg::kTileBytes);
        for (int h = 0; h < Cfg::kHalves; ++h)
          tma_load_3d(sbase + Cfg::kOffK + st * Cfg::kTileBytes + h * 16384, &mk, bar(TS_K_FULL + st), h * 64,
                      (i % p.k_tiles) * 128, unit);
      }
      if (!ok) {
        // let the copies that are still in flight land before the thread block goes away
        if (n_q > 0) mbar_wait_brief(bar(TS_Q_FULL), (n_q - 1) & 1);
        for (int x = max(0, g - Cfg::kStages); x < g; ++x)
          mbar_wait_brief(bar(TS_K_FULL + x % Cfg::kStages), (x / Cfg::kStages) & 1);
      }
    }
  } else if (warp == Cfg::kWarpIss) {
    const uint32_t idesc = umma_idesc_bf16(128, 128, false);
    bool ok = true;
    int n_q = 0, g = 0;
    for (int i = from; i < to && ok; ++i, ++g) {
      if (i == from || i % p.k_tiles == 0) ok = mbar_wait_warp(bar(TS_Q_FULL), n_q++ & 1, ab, p.err, 3101);
      const int st = g % Cfg::kStages, b = g & 1;
      if (ok) ok = mbar_wait_warp(bar(TS_K_FULL + st), (g / Cfg::kStages) & 1, ab, p.err, 3105);
      if (ok && g >= 2) ok = mbar_wait_warp(bar(TS_S_EMPTY + b), ((g >> 1) - 1) & 1, ab, p.err, 3106);
      if (!ok) break;
      tc_fence_after();
      const uint32_t kb = sbase + Cfg::kOffK + st * Cfg::kTileBytes;
      if (elect_one()) {               // one election for both products and the commits
#pragma unroll
        for (int part = 0; part < 2; ++part) {
#pragma unroll
          for (int kk = 0; kk < D / 16; ++kk) {
            const uint32_t off = (kk / 4) * 16384 + (kk % 4) * 32;
            umma_ss(tmem + b * 128, umma_smem_desc_sw128(sbase + part * Cfg::kTileBytes + off, 16, 1024),
                    umma_smem_desc_sw128(kb + off, 16, 1024), idesc, (part | kk) ? 1u : 0u);
          }
        }
        umma_commit(bar(TS_S_FULL + b));
        umma_commit(bar(TS_K_EMPTY + st));
        if ((i + 1) % p.k_tiles == 0) umma_commit(bar(TS_Q_EMPTY));
      }
      __syncwarp();
    }
  } else {
    const int b = warp >> 2, wq = warp & 3;
    const bool wide = (reinterpret_cast<uintptr_t>(p.scores) & 31) == 0;       // (rows are whole multiples of 512 bytes)
    bool ok = true;
    for (int i = from + b, f = 0; i < to; i += 2, ++f) {
      ok = mbar_wait(bar(TS_S_FULL + b), f & 1, ab, p.err, 3102);
      if (!ok) break;
      tc_fence_after();
      const int row = i / p.k_tiles, unit = row / p.q_tiles, key0 = (i - row * p.k_tiles) * 128;
      const int qb = (row - unit * p.q_tiles) * 128 + wq * 32 + lane;
      float* dst = p.scores + (size_t(unit) * p.n_blocks + qb) * p.s_stride + key0;
      const int live = p.kv_len - key0;                    // columns of this tile with a key
#pragma unroll
      for (int cc = 0; cc < 4; ++cc) {
        uint32_t r[32];
        tmem_ld32(tmem + (uint32_t(wq * 32) << 16) + b * 128 + cc * 32, r);
        tmem_ld_wait();
        if (cc == 3) {
          tc_fence_before();
          mbar_arrive(bar(TS_S_EMPTY + b));
        }
        if (live < 128) {
#pragma unroll
          for (int e = 0; e < 32; ++e)
            if (cc * 32 + e >= live) r[e] = __float_as_uint(-INFINITY);
        }
        if (qb < p.n_blocks) {
#pragma unroll
          for (int e = 0; e < 32; e += 8) {
            if (wide) {
              st_global_v8(dst + cc * 32 + e, &r[e]);
            } else {
              *reinterpret_cast<uint4*>(dst + cc * 32 + e) = make_uint4(r[e], r[e + 1], r[e + 2], r[e + 3]);
              *reinterpret_cast<uint4*>(dst + cc * 32 + e + 4) = make_uint4(r[e + 4], r[e + 5], r[e + 6], r[e + 7]);
            }
          }
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == Cfg::kWarpProd) {
    __syncwarp();
    tmem_dealloc(tmem, 256);
  }
}

// Orderable image of a float: a larger float gives a larger unsigned key.
__device__ __forceinline__ uint32_t float_order_key(float x) {
  const uint32_t u = __float_as_uint(x);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

__device__ __forceinline__ float float_of_order_key(uint32_t key) {
  return __uint_as_float((key & 0x80000000u) ? (key ^ 0x80000000u) : ~key);
}

constexpr int kSelThreads = 512;
constexpr int kSelBins = 2048;
constexpr uint32_t kSelBinSort = 64;         // entries of one bin that are ordered by counting

// Entries that the selection collects at most.  A quarter more than k leaves room for a threshold that is read off a sample
// (and 1024 for the small k, whose share of the sample is a few entries); a power of two at least k is what the sort needs.
inline int select_capacity(int k) {
  int pow2 = 2;
  while (pow2 < k) pow2 <<= 1;
  const int wide = (k + (k >> 2) + 63) & ~63;
  return wide > pow2 ? (wide > 1024 ? wide : 1024) : (pow2 > 1024 ? pow2 : 1024);
}

// grid (rows), kSelThreads threads.  Row r of `scores` has n entries (stride s_stride, a multiple of 4, rows 16-byte
// aligned).  The k largest (equal scores: smaller index first), 1 <= k <= n:
// BITS = false: their indices in descending score order to idx[r][0..k), k to cnt[r], list_stride to the slots behind.
//   Dynamic shared memory: 8 * (cap + kSelBinSort) + 2 * cap bytes.
// BITS = true: their bits set in row r of `bits` (row_words words), the others clear; what an attention step needs of a
//   selection, without the order.  Dynamic shared memory: 8 * (cap + kSelBinSort) + 4 * row_words bytes.
//
// A sample of the row, 16 of every 128 bytes, gives a score that more than k and fewer than cap entries reach -- nearly
// always; one sweep then collects those, and the count says whether it was so.  Rows where it was not go the general way
// (below), which needs the range of the keys, one to three histogram sweeps and a sweep that collects.  3072 rows of
// 32760 scores, k = 3276, means, scores and selection against the general way for all rows: 579 -> 402 us; with a NaN or one
// score far above the others 880 -> 397; half of them equal 736 -> 572, all of few values 1195 -> 1240.
// PER_SM: thread blocks that an SM's shared memory has room for.  Three leave 40 registers a thread, a few too few for the
// general way: 8192 keys of rows of equal scores, where two fit anyway, 1.67 -> 1.58 ms with the registers of two.
constexpr int kSelSmemOfThree = 66 * 1024;
template <bool BITS, int PER_SM>
__global__ void __launch_bounds__(kSelThreads, PER_SM)
topk_select_kernel(const float* scores, int s_stride, int n, int k, int k_pow2, int cap, int* idx,
                   int* cnt, int list_stride, uint32_t* bits, int row_words) {
  // (key << 32 | ~index), cap entries and room for a bin's; then cap slots, or the row's bits
  extern __shared__ unsigned long long sel[];
  __shared__ int hist[kSelBins];
  __shared__ uint32_t s_lo, s_hi, s_max;
  __shared__ int s_rem, s_ties, s_count, s_base;
  __shared__ uint32_t red_lo[kSelThreads / 32], red_hi[kSelThreads / 32];
  __shared__ int warp_tot[kSelThreads / 32];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  grid_trigger();
  grid_wait();
  const float* row = scores + size_t(blockIdx.x) * s_stride;
  const float4* row4 = reinterpret_cast<const float4*>(row);
  const int n4 = (n + 3) >> 2;
  unsigned long long* const after = sel + cap + kSelBinSort;
  uint16_t* slot = reinterpret_cast<uint16_t*>(after);
  uint32_t* row_bits = reinterpret_cast<uint32_t*>(after);

  // One sweep over the row, four 16-byte loads in flight per thread; f(key, index, live) per entry.
  // The trip count is the same for every thread, so f may use full-warp collectives.
  auto sweep = [&](auto&& f) {
    for (int base = 0; base < n4; base += 4 * kSelThreads) {
      float4 v[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int j = base + u * kSelThreads + tid;
        v[u] = (j < n4) ? row4[j] : make_float4(0.f, 0.f, 0.f, 0.f);
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int j = base + u * kSelThreads + tid;
        const float x[4] = {v[u].x, v[u].y, v[u].z, v[u].w};
#pragma unroll
        for (int e = 0; e < 4; ++e) f(float_order_key(x[e]), 4 * j + e, j < n4 && 4 * j + e < n);
      }
    }
  };
  // smallest and largest key over the block -> s_lo, s_hi
  auto key_range = [&](uint32_t kmin, uint32_t kmax) {
    kmin = __reduce_min_sync(0xffffffffu, kmin);
    kmax = __reduce_max_sync(0xffffffffu, kmax);
    if (lane == 0) { red_lo[warp] = kmin; red_hi[warp] = kmax; }
    __syncthreads();
    if (tid == 0) {
      uint32_t a = red_lo[0], b = red_hi[0];
      for (int w = 1; w < kSelThreads / 32; ++w) { a = min(a, red_lo[w]); b = max(b, red_hi[w]); }
      s_lo = a;
      s_hi = b;
    }
    __syncthreads();
  };
  auto clear_hist = [&]() {
    for (int i = tid; i < kSelBins; i += kSelThreads) hist[i] = 0;
  };
  // Exclusive sums over the bins into hist, four bins per thread; returns the fullest bin's count.
  auto scan_hist = [&]() -> uint32_t {
    static_assert(kSelBins == 4 * kSelThreads, "four bins per thread");
    int c[4], sum = 0, most = 0;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      c[u] = hist[4 * tid + u];
      sum += c[u];
      most = max(most, c[u]);
    }
    int incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += t;
    }
    most = __reduce_max_sync(0xffffffffu, most);
    if (lane == 31) warp_tot[warp] = incl;
    if (lane == 0) red_hi[warp] = uint32_t(most);
    __syncthreads();
    int start = incl - sum;
    uint32_t fullest = 0;
#pragma unroll
    for (int w = 0; w < kSelThreads / 32; ++w) {
      if (w < warp) start += warp_tot[w];
      fullest = max(fullest, red_hi[w]);
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      hist[4 * tid + u] = start;
      start += c[u];
    }
    __syncthreads();
    return fullest;
  };
  // bins of equal score width from f_hi down to f_lo; false where the scores do not spread over a finite range (f_hi == f_lo
  // gives an infinite factor, so does a range under about 1e-35, an infinite score a zero or NaN)
  float f_hi = 0.f, to_bin = 0.f;
  auto set_bins = [&](uint32_t key_hi, uint32_t key_lo) -> bool {
    f_hi = float_of_order_key(key_hi);
    to_bin = float(kSelBins - 1) / (f_hi - float_of_order_key(key_lo));
    return to_bin > 0.f && to_bin < 1e30f;
  };
  // (scores above f_hi and NaN go to the first bin)
  auto bin_of_key = [&](uint32_t key) -> int {
    return int(fminf(fmaxf((f_hi - float_of_order_key(key)) * to_bin, 0.f), float(kSelBins - 1)));
  };

  // The k largest of the m >= k entries in sel, whose keys are key_lo or more and most of them key_hi or less, by counting: the entries are counted into
  // 2048 bins of equal width over their range of scores (a monotone map, so a larger bin holds smaller scores), every
  // entry gets a slot in its bin, and inside a bin -- a few entries -- an entry's place is the number of larger ones.
  // Five barriers where a bitonic sort of 4096 entries takes 78 passes: 3276 of 32760 keys for 3072 rows, the whole
  // selection 1.017 -> 0.569 ms (8192 keys 1.864 -> 1.001 ms).  False, and nothing written, for scores that pile up in a
  // few bins (equal or infinite ones, or one far above all others), where counting inside the bins would be quadratic:
  // with kSelBinSort = 256 one score at 30 deviations takes 3.2 ms at 8192 keys, by the sort 1.55.
  auto finish_by_counting = [&](int m, uint32_t key_hi, uint32_t key_lo) -> bool {
    if (!set_bins(key_hi, key_lo)) return false;
    clear_hist();
    if (tid == 0) s_count = 0;
    __syncthreads();
    for (int i = tid; i < m; i += kSelThreads) atomicAdd(&hist[bin_of_key(uint32_t(sel[i] >> 32))], 1);
    __syncthreads();
    if (scan_hist() > kSelBinSort) return false;
    // hist[b] is the start of bin b
    if constexpr (BITS) {
      for (int i = tid; i < row_words; i += kSelThreads) row_bits[i] = 0u;
      __syncthreads();
      auto set_bit = [&](unsigned long long e) {
        const uint32_t i = ~uint32_t(e & 0xffffffffull);
        atomicOr(&row_bits[i >> 5], 1u << (i & 31));
      };
      // bins that end at k or before are taken whole, the entries of the one that k falls into are compared
      unsigned long long* edge = sel + cap;
      for (int i = tid; i < m; i += kSelThreads) {
        const unsigned long long e = sel[i];
        const int b = bin_of_key(uint32_t(e >> 32));
        if ((b + 1 < kSelBins ? hist[b + 1] : m) <= k) set_bit(e);
        else if (hist[b] < k) edge[atomicAdd(&s_count, 1)] = e;
      }
      __syncthreads();
      const int c = s_count;
      if (tid < c) {
        const unsigned long long e = edge[tid];
        int place = hist[bin_of_key(uint32_t(e >> 32))];
        for (int j = 0; j < c; ++j) place += edge[j] > e ? 1 : 0;
        if (place < k) set_bit(e);
      }
      __syncthreads();
      uint32_t* dst = bits + size_t(blockIdx.x) * row_words;
      for (int i = tid; i < row_words; i += kSelThreads) dst[i] = row_bits[i];
    } else {
      for (int i = tid; i < m; i += kSelThreads) slot[atomicAdd(&hist[bin_of_key(uint32_t(sel[i] >> 32))], 1)] = uint16_t(i);
      __syncthreads();
      // hist[b] is now the end of bin b, which is where bin b + 1 starts
      int* dst = idx + size_t(blockIdx.x) * list_stride;
      for (int i = tid; i < m; i += kSelThreads) {
        const unsigned long long e = sel[i];
        const int b = bin_of_key(uint32_t(e >> 32)), s0 = b ? hist[b - 1] : 0, s1 = hist[b];
        int place = s0;
        for (int j = s0; j < s1; ++j) place += sel[slot[j]] > e ? 1 : 0;
        if (place < k) dst[place] = int(~uint32_t(e & 0xffffffffull));
      }
      for (int i = k + tid; i < list_stride; i += kSelThreads) dst[i] = list_stride;
      if (tid == 0) cnt[blockIdx.x] = k;
    }
    return true;
  };

  int sort_n = 0;                                        // entries of sel to sort, a power of two (zeros fill up); none yet
  // ---- the short way
  {
    // The sample: of every 32 entries the four at a place that changes from one to the next, so that keys which differ by
    // their place in the rows of an image, of a multiple of 32 keys, are like their sample.  A fixed place: 3072 rows of
    // 32760 scores, k = 3276, where 4 of every 32 keys stand out 648 us for the whole selection instead of 428.
    const int m4 = n >> 5;                                 // float4s of the sample
    uint32_t kmin = 0xffffffffu, kmax = 0u;
    auto sample = [&](auto&& f) {
      for (int i = tid; i < m4; i += kSelThreads) {
        const float4 v = row4[8 * i + ((uint32_t(i) * 0x9E3779B1u) >> 29)];
        const float x[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int e = 0; e < 4; ++e) f(float_order_key(x[e]));
      }
    };
    sample([&](uint32_t key) {
      kmin = min(kmin, key);
      kmax = max(kmax, key);
    });
    key_range(kmin, kmax);
    const uint32_t lo_key = s_lo, hi_key = s_hi;
    const int m = 4 * m4;
    // the sample's rank of a score that (k + cap) / 2 entries of the row reach
    const int rank = int((long long)(k + cap) * m / (2 * n));
    if (rank >= 1 && rank < m && set_bins(hi_key, lo_key)) {
      clear_hist();
      if (tid == 0) { s_count = 0; s_rem = kSelBins; }
      __syncthreads();
      sample([&](uint32_t key) { atomicAdd(&hist[bin_of_key(key)], 1); });
      __syncthreads();
      scan_hist();
      // the first bin that starts at or past that rank: its upper edge is the threshold, unless equal scores make it
      // reach more entries than there is room for
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int b = 4 * tid + u;
        if (b > 0 && hist[b] >= rank && hist[b - 1] < rank && (long long)hist[b] * n <= (long long)cap * m) s_rem = b;
      }
      __syncthreads();
      if (s_rem < kSelBins) {
        const uint32_t from = float_order_key(f_hi - float(s_rem) / to_bin);
        // reach(x): the score counts.  A threshold above zero is compared as the integer that its bits are (the larger of two
        // positive floats, NaN included, is the larger integer, and negative ones are negative integers): one instruction
        // an entry where the order-preserving image takes four.
        auto collect = [&](auto&& reach) {
          for (int base = 0; base < n4; base += 4 * kSelThreads) {
            float4 v[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
              const int j = base + u * kSelThreads + tid;
              v[u] = (j < n4) ? row4[j] : make_float4(0.f, 0.f, 0.f, 0.f);
            }
            uint32_t take = 0u;
#pragma unroll
            for (int u = 0; u < 4; ++u) {
              const float x[4] = {v[u].x, v[u].y, v[u].z, v[u].w};
#pragma unroll
              for (int e = 0; e < 4; ++e)
                if (reach(x[e])) take |= 1u << (4 * u + e);
            }
            if (base + 4 * kSelThreads > n >> 2) {           // the row ends here: entries past it do not count
#pragma unroll
              for (int u = 0; u < 4; ++u) {
                const int left = n - 4 * (base + u * kSelThreads + tid);
                if (left < 4) take &= ~((15u << (4 * u)) & (left <= 0 ? ~0u : ~((1u << (4 * u + left)) - 1u)));
              }
            }
            const int c = __popc(take);
            int incl = c;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
              const int t = __shfl_up_sync(0xffffffffu, incl, o);
              if (lane >= o) incl += t;
            }
            int at = 0;
            if (lane == 31 && incl > 0) at = atomicAdd(&s_count, incl);
            at = __shfl_sync(0xffffffffu, at, 31) + incl - c;
#pragma unroll
            for (int u = 0; u < 4; ++u) {
              const float x[4] = {v[u].x, v[u].y, v[u].z, v[u].w};
#pragma unroll
              for (int e = 0; e < 4; ++e) {
                if ((take >> (4 * u + e)) & 1u) {
                  if (at < cap)
                    sel[at] = (static_cast<unsigned long long>(float_order_key(x[e])) << 32) |
                              uint32_t(~uint32_t(4 * (base + u * kSelThreads + tid) + e));
                  ++at;
                }
              }
            }
          }
        };
        if (from > 0x80000000u) {
          const int limit = int(from & 0x7fffffffu);
          collect([&](float x) { return __float_as_int(x) >= limit; });
        } else {
          collect([&](float x) { return float_order_key(x) >= from; });
        }
        __syncthreads();
        const int got = s_count;
        __syncthreads();
        if (got >= k && got <= cap) {
          // counted up to the sample's largest score: the few above it, NaN among them, share a bin
          if (finish_by_counting(got, hi_key, from)) return;
          int size = 2;
          while (size < got) size <<= 1;
          if (size <= cap) {
            for (int i = got + tid; i < size; i += kSelThreads) sel[i] = 0ull;
            sort_n = size;
          }
        }
      }
    }
    __syncthreads();
  }

  // ---- The general way.  Every sweep reads the row from global memory (L2 after the first; keeping the row in shared
  // memory instead allows one thread block per SM only and measured slower).  Selection works on the order-preserving
  // unsigned image of the scores.  A first sweep finds the smallest and largest key of the row; each following sweep
  // histograms the keys of the current interval into 2048 equal bins (a plain byte-wise radix would put almost every score
  // of a row into two or three bins of its leading byte and serialise the shared-memory counters), picks the bin that
  // holds the k-th largest and narrows the interval to it, until the bin and everything above it fit the sort buffer
  // (usually after one histogram sweep) or the bins are one key wide.
  if (sort_n == 0) {
    // ---- key range of the row
    uint32_t kmin = 0xffffffffu, kmax = 0u;
    sweep([&](uint32_t key, int, bool live) {
      if (live) {
        kmin = min(kmin, key);
        kmax = max(kmax, key);
      }
    });
    key_range(kmin, kmax);
    if (tid == 0) {
      s_max = s_hi;
      s_rem = k;
    }
    __syncthreads();

    // ---- narrow [lo, hi] around the k-th largest key.  hi - lo < 2^shift after a sweep, so shift goes from 21 at most to
    // 10 to 0: three sweeps at most.
    while (true) {
      const uint32_t lo = s_lo, hi = s_hi;
      const int rem = s_rem;
      const uint32_t width = hi - lo;                                    // keys in the interval - 1
      const int shift = max(0, (32 - __clz(width | 1u)) - 11);           // (hi - lo) >> shift < 2048
      for (int i = tid; i < kSelBins; i += kSelThreads) hist[i] = 0;
      __syncthreads();
      sweep([&](uint32_t key, int, bool live) {
        if (live && key >= lo && key <= hi) atomicAdd(&hist[(key - lo) >> shift], 1);
      });
      __syncthreads();
      if (warp == 0) {
        // lane L owns the 64 bins [2048 - 64 (L + 1), 2048 - 64 L): lane 0 holds the largest keys
        constexpr int kPer = kSelBins / 32;
        const int b0 = kSelBins - kPer * (lane + 1);
        int mine = 0;
        for (int b = 0; b < kPer; ++b) mine += hist[b0 + b];
        int incl = mine;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int t = __shfl_up_sync(0xffffffffu, incl, o);
          if (lane >= o) incl += t;
        }
        const bool here = incl >= rem && incl - mine < rem;              // exactly one lane
        if (here) {
          int r = rem - (incl - mine), b = kPer - 1;
          for (; b > 0; --b) {
            if (hist[b0 + b] >= r) break;
            r -= hist[b0 + b];
          }
          const uint32_t nlo = lo + (uint32_t(b0 + b) << shift);
          s_lo = nlo;
          s_hi = nlo + min(hi - nlo, (1u << shift) - 1u);          // (the keys of NaNs reach 2^32 - 1: no wrap)
          s_rem = r;
          s_ties = hist[b0 + b];
        }
      }
      __syncthreads();
      // stop as soon as everything from the chosen bin upwards fits the sort buffer: the sort then
      // orders the bin's entries too and the first k sorted entries are the answer
      if (shift == 0 || (k - s_rem) + s_ties <= k_pow2) break;
    }
    const uint32_t kth = s_lo;                             // lowest key taken; s_rem of the s_ties entries in
                                                           // [kth, s_hi] are needed (s_hi == kth after a full narrowing)
    const int rem = s_rem, n_gt = k - rem;
    __syncthreads();

    if (tid == 0) { s_count = 0; s_base = 0; }
    for (int i = tid; i < k_pow2; i += kSelThreads) sel[i] = 0ull;
    __syncthreads();
    if (n_gt + s_ties <= k_pow2) {
      // ---- common case: everything >= kth fits the sort buffer; the sort puts ties in index order.
      // One shared-counter update per warp and sweep slot.
      sweep([&](uint32_t key, int i, bool live) {
        const bool take = live && key >= kth;
        const uint32_t bal = __ballot_sync(0xffffffffu, take);
        if (bal) {
          int base = 0;
          if (lane == __ffs(bal) - 1) base = atomicAdd(&s_count, __popc(bal));
          base = __shfl_sync(0xffffffffu, base, __ffs(bal) - 1);
          if (take)
            sel[base + __popc(bal & ((1u << lane) - 1u))] =
                (static_cast<unsigned long long>(key) << 32) | uint32_t(~uint32_t(i));
        }
      });
    } else {
      // ---- many ties at the k-th key: entries above it in any order, then the first `rem` ties by index
      for (int i0 = 0; i0 < n; i0 += kSelThreads) {
        const int i = i0 + tid;
        const uint32_t key = (i < n) ? float_order_key(row[i]) : 0u;
        if (i < n && key > kth) {
          const int pos = atomicAdd(&s_count, 1);
          sel[pos] = (static_cast<unsigned long long>(key) << 32) | uint32_t(~uint32_t(i));
        }
        const int tie = (i < n && key == kth) ? 1 : 0;
        const uint32_t bal = __ballot_sync(0xffffffffu, tie);
        if (lane == 0) warp_tot[warp] = __popc(bal);
        __syncthreads();
        int off = s_base;
        for (int w = 0; w < warp; ++w) off += warp_tot[w];
        off += __popc(bal & ((1u << lane) - 1u));
        if (tie && off < rem)
          sel[n_gt + off] = (static_cast<unsigned long long>(key) << 32) | uint32_t(~uint32_t(i));
        __syncthreads();
        if (tid == kSelThreads - 1) s_base = off + tie;
        __syncthreads();
      }
    }
    __syncthreads();

    const int m = (n_gt + s_ties <= k_pow2) ? n_gt + s_ties : k;
    const uint32_t key_top = s_max;
    if (finish_by_counting(m, key_top, kth)) return;
    __syncthreads();
    sort_n = k_pow2;
  }

  // ---- bitonic sort, descending: the first k entries are the answer.  The passes of strides up to 32 stay inside groups
  // of 64 entries: a warp takes a group through all of them in registers, two entries a lane, and only the passes
  // of wider strides go through shared memory with a block barrier each (28 of 91 at 8192 entries).  Selections that end
  // here pay for the histogram above too; with every pass through shared memory that made them slower than the sort
  // alone: half of the scores equal, 3276 keys 1.234 -> 1.251 ms, now 1.156; 8192 keys 1.906 -> 2.102, now 1.826; one
  // score at 30 deviations 1.017 -> 1.027, now 0.849, and 1.893 -> 1.990, now 1.550.
  auto in_group = [&](int size_from, int size_to) {        // the passes of these sizes whose strides are 32 or less
    for (int g = warp * 64; g < sort_n; g += (kSelThreads / 32) * 64) {
      unsigned long long x[2];
#pragma unroll
      for (int h = 0; h < 2; ++h) x[h] = (g + 32 * h + lane < sort_n) ? sel[g + 32 * h + lane] : 0ull;
      for (int size = size_from; size <= size_to; size <<= 1) {
        if (size >= 64) {
          const bool desc = (g & size) == 0;
          const unsigned long long a = x[0], b = x[1];
          x[0] = ((a < b) == desc) ? b : a;
          x[1] = ((a < b) == desc) ? a : b;
        }
        for (int stride = min(size, 32) >> 1; stride > 0; stride >>= 1) {
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const unsigned long long y = __shfl_xor_sync(0xffffffffu, x[h], stride);
            const bool desc = ((g + 32 * h + lane) & size) == 0, upper = (lane & stride) != 0;
            x[h] = ((x[h] < y) == (desc != upper)) ? y : x[h];
          }
        }
      }
#pragma unroll
      for (int h = 0; h < 2; ++h)
        if (g + 32 * h + lane < sort_n) sel[g + 32 * h + lane] = x[h];
    }
    __syncthreads();
  };
  in_group(2, 64);                                         // (entries past the end of a short list count as zeros, the smallest)
  for (int size = 128; size <= sort_n; size <<= 1) {
    for (int stride = size >> 1; stride > 32; stride >>= 1) {
      for (int t = tid; t < (sort_n >> 1); t += kSelThreads) {
        const int lo = 2 * t - (t & (stride - 1)), hi = lo + stride;
        const bool desc = (lo & size) == 0;
        const unsigned long long a = sel[lo], b = sel[hi];
        if ((a < b) == desc) {
          sel[lo] = b;
          sel[hi] = a;
        }
      }
      __syncthreads();
    }
    in_group(size, size);
  }
  if constexpr (BITS) {
    for (int i = tid; i < row_words; i += kSelThreads) row_bits[i] = 0u;
    __syncthreads();
    for (int i = tid; i < k; i += kSelThreads) {
      const uint32_t key = ~uint32_t(sel[i] & 0xffffffffull);
      atomicOr(&row_bits[key >> 5], 1u << (key & 31));
    }
    __syncthreads();
    uint32_t* dst = bits + size_t(blockIdx.x) * row_words;
    for (int i = tid; i < row_words; i += kSelThreads) dst[i] = row_bits[i];
  } else {
    int* dst = idx + size_t(blockIdx.x) * list_stride;
    for (int i = tid; i < k; i += kSelThreads) dst[i] = int(~uint32_t(sel[i] & 0xffffffffull));
    for (int i = k + tid; i < list_stride; i += kSelThreads) dst[i] = list_stride;
    if (tid == 0) cnt[blockIdx.x] = k;
  }
}

}  // namespace fg
