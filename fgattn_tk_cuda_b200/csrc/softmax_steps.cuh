// Per-thread softmax steps shared by the dense and the block-sparse kernels.  A thread owns one
// query row (one TMEM lane) and sees one 128-key score tile as two 64-key halves; `valid0` and
// `valid1` give the number of live columns in each half (0..64), the rest is masked out.
#pragma once
#include "sm100_ptx.cuh"

namespace fg {

struct OnlineState {
  float m_used;   // running maximum in the scaled log2 domain (s * c); may lag the true one by < 8
  float m_true;   // exact running raw maximum
  float l;        // running denominator relative to m_used
};

// exponent (log2 domain, relative to the running maximum) below which a whole 32-column quarter
// is treated as zero by softmax_online_step
constexpr float kSkipLog2 = -40.0f;

__device__ __forceinline__ void online_init(OnlineState& st) {
  st.m_used = -1.0e30f;
  st.m_true = -INFINITY;
  st.l = 0.f;
}

// Multiplies one row of the accumulator (D fp32 columns at o_addr) by alpha.  Nothing may still be adding to it.  Where
// the query tile has one score buffer, the commit that published its scores covers its previous P*V product too.  With
// rotating scores they come while that product may still be running: the caller waits for it first.
template <int D>
__device__ __forceinline__ void rescale_accumulator(uint32_t o_addr, float alpha) {
#pragma unroll
  for (int cc = 0; cc < D / 32; ++cc) {
    uint32_t o[32];
    tmem_ld32(o_addr + cc * 32, o);
    tmem_ld_wait();
#pragma unroll
    for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
    tmem_st32(o_addr + cc * 32, o);
  }
}

// Online softmax over one score tile.
//   s_addr : TMEM address (lane already folded in) of the 128 fp32 score columns
//   p_addr : where the 64 packed-bf16 probability columns go (WRITE_P)
//   o_addr : the row's D fp32 output accumulator columns (rescaled in place when the maximum grows)
// Returns the raw maxima of the two 64-key halves through mx0 / mx1.
//   colmask: optional 128-bit column mask (4 words, bit set = live column) applied on top
//   POLY   : of every eight pairs of columns, how many compute their exponentials on the FMA pipe
//            (ex2_poly2) instead of the MUFU, which is the busiest unit of these kernels.  Measured with
//            L2 flushed between calls: 2 of 8 with P*V (C2 0.245 -> 0.232 ms, C4 5.33 -> 5.11 ms, C3 within
//            2 %), 3 of 8 for the max / denominator pass (C3 2.49 -> 2.38 ms, C4 3.94 -> 3.45 ms); 4 of 8 is
//            slower again: the polynomial costs ten issue slots per pair against two
//   SKIP   : quarters of 32 columns that are negligible in all rows of a warp (kSkipLog2) take no exponentials.  The
//            maximum passes over NaN, so a NaN score among negligible ones is skipped with them, and an infinite V row
//            then meets a probability of zero instead of a tiny one.  Without: only quarters that the mask leaves out.
//   quiet  : called before the accumulator is touched (waits for a product that may still be adding to it)
//   loaded : called when the scores are in registers
struct NoWait {
  __device__ __forceinline__ void operator()() const {}
};
template <int D, bool WRITE_P, int POLY = (WRITE_P ? 2 : 3), bool SKIP = true, class Quiet = NoWait, class Loaded = NoWait>
__device__ __forceinline__ void softmax_online_step(uint32_t s_addr, uint32_t p_addr, uint32_t o_addr, int valid0,
                                                    int valid1, float c, bool first, OnlineState& st, float& mx0,
                                                    float& mx1, const uint32_t* colmask = nullptr,
                                                    Quiet quiet = Quiet(), Loaded loaded = Loaded()) {
  uint32_t r[128];
#pragma unroll
  for (int cc = 0; cc < 4; ++cc) tmem_ld32(s_addr + cc * 32, *reinterpret_cast<uint32_t(*)[32]>(&r[cc * 32]));
  tmem_ld_wait();
  loaded();
  if (valid0 < 64 || valid1 < 64) {
#pragma unroll
    for (int i = 0; i < 64; ++i) {
      if (i >= valid0) r[i] = __float_as_uint(-INFINITY);
      if (i >= valid1) r[64 + i] = __float_as_uint(-INFINITY);
    }
  }
  if (colmask != nullptr) {
#pragma unroll
    for (int w = 0; w < 4; ++w) {
      const uint32_t mw = colmask[w];
      if (mw != 0xffffffffu) {
#pragma unroll
        for (int i = 0; i < 32; ++i)
          if (!((mw >> i) & 1u)) r[w * 32 + i] = __float_as_uint(-INFINITY);
      }
    }
  }
  // maxima of the four 32-column quarters (four independent chains)
  float qmax[4];
#pragma unroll
  for (int w = 0; w < 4; ++w) qmax[w] = __uint_as_float(r[w * 32]);
#pragma unroll
  for (int i = 1; i < 32; ++i) {
#pragma unroll
    for (int w = 0; w < 4; ++w) qmax[w] = fmaxf(qmax[w], __uint_as_float(r[w * 32 + i]));
  }
  mx0 = fmaxf(qmax[0], qmax[1]);
  mx1 = fmaxf(qmax[2], qmax[3]);
  const float mx = fmaxf(mx0, mx1);
  st.m_true = fmaxf(st.m_true, mx);
  const float ms = mx * c;
  const bool grow = ms > st.m_used + 8.0f;
  if (__any_sync(0xffffffffu, grow)) {
    const float alpha = grow ? ex2(st.m_used - ms) : 1.0f;
    if (grow) st.m_used = ms;
    st.l *= alpha;
    if (WRITE_P && !first) {
      quiet();
      rescale_accumulator<D>(o_addr, alpha);
    }
  }
  float sum0 = 0.f, sum1 = 0.f;
  const float neg_m = -st.m_used;
#pragma unroll
  for (int w = 0; w < 4; ++w) {
    // A quarter whose largest exponent is below kSkipLog2 for every row of the warp contributes
    // less than 2^-40 per entry relative to the running maximum -- under one fp32 ulp of the
    // denominator and of the output even summed over a whole row -- so its exponentials are
    // skipped and its probabilities are exact zeros.
    const bool skip = SKIP ? __all_sync(0xffffffffu, fmaf(qmax[w], c, neg_m) < kSkipLog2)
                           : colmask != nullptr && colmask[w] == 0u;
    if (skip) {
      if (WRITE_P) {
#pragma unroll
        for (int i = 0; i < 16; ++i) r[w * 16 + i] = 0u;
      }
      continue;
    }
#pragma unroll
    for (int i = w * 32; i < w * 32 + 32; i += 2) {
      float p0, p1;
      if constexpr (POLY > 0) {
        // packed scale-and-shift; the pairs that take the FMA-pipe exponential are spread evenly
        const uint64_t x2 = f2_fma(f2_pack(__uint_as_float(r[i]), __uint_as_float(r[i + 1])), f2_pack(c, c),
                                   f2_pack(neg_m, neg_m));
        if ((((i >> 1) & 7) * POLY) % 8 < POLY) {
          ex2_poly2(x2, p0, p1);
        } else {
          float x0, x1;
          f2_unpack(x2, x0, x1);
          p0 = ex2(x0);
          p1 = ex2(x1);
        }
      } else {
        p0 = ex2(fmaf(__uint_as_float(r[i]), c, neg_m));
        p1 = ex2(fmaf(__uint_as_float(r[i + 1]), c, neg_m));
      }
      sum0 += p0;
      sum1 += p1;
      if (WRITE_P) r[i >> 1] = pack_bf16(p0, p1);
    }
  }
  st.l += sum0 + sum1;
  if (WRITE_P) {
#pragma unroll
    for (int cc = 0; cc < 4; ++cc) tmem_st16(p_addr + cc * 16, *reinterpret_cast<uint32_t(*)[16]>(&r[cc * 16]));
    tmem_st_wait();
  }
}

// Maximum of 32 scores (two chains of the three-input form).
__device__ __forceinline__ float quarter_max(const uint32_t (&r)[32]) {
  float a = __uint_as_float(r[0]), b = __uint_as_float(r[1]);
#pragma unroll
  for (int i = 2; i < 30; i += 4) {
    a = max3(a, __uint_as_float(r[i]), __uint_as_float(r[i + 1]));
    b = max3(b, __uint_as_float(r[i + 2]), __uint_as_float(r[i + 3]));
  }
  return fmaxf(max3(a, __uint_as_float(r[30]), __uint_as_float(r[31])), b);
}

// Probabilities of one 32-column quarter against the fixed offset -neg_m, packed to bf16 over r[0..15];
// sum2 takes the even and the odd columns' sums.  POLY and SKIP as in softmax_online_step.
template <int POLY, bool SKIP>
__device__ __forceinline__ void quarter_probs(uint32_t (&r)[32], float qmax, float c, float neg_m, uint64_t& sum2) {
  if (SKIP && __all_sync(0xffffffffu, fmaf(qmax, c, neg_m) < kSkipLog2)) {
#pragma unroll
    for (int i = 0; i < 16; ++i) r[i] = 0u;
    return;
  }
#pragma unroll
  for (int i = 0; i < 32; i += 2) {
    float p0, p1;
    const uint64_t x2 = f2_fma(f2_pack(__uint_as_float(r[i]), __uint_as_float(r[i + 1])), f2_pack(c, c),
                               f2_pack(neg_m, neg_m));
    if ((((i >> 1) & 7) * POLY) % 8 < POLY) {
      ex2_poly2(x2, p0, p1);
    } else {
      float x0, x1;
      f2_unpack(x2, x0, x1);
      p0 = ex2(x0);
      p1 = ex2(x1);
    }
    sum2 = f2_add(sum2, f2_pack(p0, p1));
    r[i >> 1] = pack_bf16(p0, p1);
  }
}

// softmax_online_step with P over a whole, unmasked 128-key score tile that is not the first of its item.  The
// offset in use may lag the running maximum by up to 2^8, so on most inputs it hardly ever moves: the exponentials start
// against the offset as it stands, before the tile's maximum is known and while three quarters of the scores are still on
// their way from tensor memory.  Where some row of the warp turns out to need a larger offset, nothing has been
// written yet: that first quarter is loaded again and the probabilities of all quarters taken against the new one.  The
// results are those of softmax_online_step bit for bit (backwards the row sums add up in another order).  Taken by the
// dense kernel at D = 64, where the softmax bounds a step ((2, 16, 4096, 64), i.i.d. normal q and k, 0.224 -> 0.217 ms), and by
// the full steps of the token lists, whose softmax is a link of a slot's chain, at both head dimensions.  The dense kernel at
// D = 128 is level to 2.5 % slower with it (32768 x 512 keys 0.374 -> 0.384 ms): two products and their hand-offs pace a step.
// `backwards` (warp-uniform): the quarters are taken last to first.  Only the first one taken is ever loaded again, so the
// columns of the other half of the tile may be overwritten as soon as `loaded` has been called.
template <int D, int POLY = 2, bool SKIP = true, class Quiet = NoWait, class Loaded = NoWait>
__device__ __forceinline__ void softmax_steady_step(uint32_t s_addr, uint32_t p_addr, uint32_t o_addr, float c,
                                                    OnlineState& st, float& mx0, float& mx1, Quiet quiet = Quiet(),
                                                    Loaded loaded = Loaded(), bool backwards = false) {
  uint32_t r[4][32];
  float qm[4];
  const float neg_m = -st.m_used;
  uint64_t sum2 = f2_pack(0.f, 0.f);
  const uint32_t s_first = s_addr + (backwards ? 96 : 0), p_first = p_addr + (backwards ? 48 : 0);
  const int ds = backwards ? -32 : 32, dp = backwards ? -16 : 16;
  tmem_ld32(s_first, r[0]);
  tmem_ld_wait_for(r[0]);
#pragma unroll
  for (int w = 1; w < 4; ++w) tmem_ld32(s_first + w * ds, r[w]);
  qm[0] = quarter_max(r[0]);
  quarter_probs<POLY, SKIP>(r[0], qm[0], c, neg_m, sum2);
#pragma unroll
  for (int w = 1; w < 4; ++w) {
    tmem_ld_wait_for(r[w]);
    qm[w] = quarter_max(r[w]);
  }
  loaded();
  const float lo = fmaxf(qm[0], qm[1]), hi = fmaxf(qm[2], qm[3]);
  mx0 = backwards ? hi : lo;
  mx1 = backwards ? lo : hi;
  const float mx = fmaxf(mx0, mx1);
  st.m_true = fmaxf(st.m_true, mx);
  auto finish = [&](float off, int from) {
#pragma unroll
    for (int w = 0; w < 4; ++w) {
      if (w >= from) quarter_probs<POLY, SKIP>(r[w], qm[w], c, off, sum2);
      tmem_st16(p_first + w * dp, *reinterpret_cast<uint32_t(*)[16]>(&r[w][0]));
    }
    float sum0, sum1;
    f2_unpack(sum2, sum0, sum1);
    st.l += sum0 + sum1;
    tmem_st_wait();
  };
  const float ms = mx * c;
  const bool grow = ms > st.m_used + 8.0f;
  if (__any_sync(0xffffffffu, grow)) {
    const float alpha = grow ? ex2(st.m_used - ms) : 1.0f;
    if (grow) st.m_used = ms;
    st.l *= alpha;
    quiet();
    rescale_accumulator<D>(o_addr, alpha);
    tmem_ld32(s_first, r[0]);
    tmem_ld_wait_for(r[0]);
    sum2 = f2_pack(0.f, 0.f);
    finish(-st.m_used, 0);
    return;
  }
  finish(neg_m, 1);
}

// Write one row of the fp32 accumulator (D columns at o_addr) as bf16, scaled by `inv`.
template <int D>
__device__ __forceinline__ void store_o_row(uint32_t o_addr, __nv_bfloat16* orow, float inv, bool in_range) {
#pragma unroll
  for (int cc = 0; cc < D / 32; ++cc) {
    uint32_t o[32];
    tmem_ld32(o_addr + cc * 32, o);
    tmem_ld_wait();
    if (in_range) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        uint4 v;
        v.x = pack_bf16(__uint_as_float(o[8 * i + 0]) * inv, __uint_as_float(o[8 * i + 1]) * inv);
        v.y = pack_bf16(__uint_as_float(o[8 * i + 2]) * inv, __uint_as_float(o[8 * i + 3]) * inv);
        v.z = pack_bf16(__uint_as_float(o[8 * i + 4]) * inv, __uint_as_float(o[8 * i + 5]) * inv);
        v.w = pack_bf16(__uint_as_float(o[8 * i + 6]) * inv, __uint_as_float(o[8 * i + 7]) * inv);
        *reinterpret_cast<uint4*>(orow + cc * 32 + i * 8) = v;
      }
    }
  }
}

// The same for the 32 rows of a warp at once, through shared memory and the TMA unit: `stage` is the warp's own
// 4 KiB buffer (1024-byte aligned, 32 rows of 128 bytes, 128-byte swizzle), `mo` the output's map with a box of 64
// columns by 32 rows, which also drops the rows past the end of the sequence.  A row-per-thread store touches 32
// cache lines per instruction, D / 8 instructions a row; here the copies leave as whole lines, asynchronously.
// `live`: the warp has a row inside the sequence.  40 heads of 32768 rows against 512 keys, D = 128 (an item is four
// key tiles long there, so that the output weighs): 0.377 -> 0.341 ms; leaving the stores out altogether gave 0.320.
template <int D>
__device__ __forceinline__ void store_o_warp(uint32_t o_addr, uint32_t stage, const CUtensorMap* mo, float inv, int row0,
                                             int unit, bool live, int lane) {
#pragma unroll
  for (int h = 0; h < D / 64; ++h) {
    uint32_t o[2][32];
    tmem_ld32(o_addr + h * 64, o[0]);
    tmem_ld32(o_addr + h * 64 + 32, o[1]);
    tmem_ld_wait_for(o[0]);
    tmem_ld_wait_for(o[1]);
    if (lane == 0) bulk_wait_read();             // the copy before this one has left the buffer
    __syncwarp();
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const uint32_t(&x)[32] = o[i / 4];
      const int e = (i & 3) * 8;
      uint32_t w[4];
#pragma unroll
      for (int u = 0; u < 4; ++u)
        w[u] = pack_bf16(__uint_as_float(x[e + 2 * u]) * inv, __uint_as_float(x[e + 2 * u + 1]) * inv);
      st_shared_v4(stage + sw128_offset(lane, i), w[0], w[1], w[2], w[3]);
    }
    fence_proxy_async_smem();
    __syncwarp();
    if (lane == 0 && live) {
      tma_store_3d(mo, stage, h * 64, row0, unit);
      bulk_commit();
    }
  }
}

}  // namespace fg
