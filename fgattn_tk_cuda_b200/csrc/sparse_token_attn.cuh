// Sparse attention over key-TOKEN lists at the reference granularity (128-row query blocks).
// For each query block the listed K/V rows are gathered 128 at a time into swizzled shared-memory
// tiles (16-byte cp.async per chunk, whole rows per warp-wide copy, seven gather warps), and the flash-attention step over the
// gathered keys runs on tcgen05 with an online (renormalising) softmax.  A CTA runs two query
// blocks ("slots") against one tensor pipe; their K/V tiles share one ring in consumption order.
// List entries >= the number of key rows, and slots past the count, are masked out.
#pragma once
#include "sm100_ptx.cuh"
#include "softmax_steps.cuh"

namespace fg {

struct TokenParams {
  __nv_bfloat16* o;
  const __nv_bfloat16* k;
  const __nv_bfloat16* v;
  const int* kv_idx;        // [BH, nqb128, mask_stride]
  const int* kv_cnt;        // [BH, nqb128]
  int* err;
  int S, S_kv, nqb, mask_stride;   // query rows, rows of k / v per head
  // thread block i works on item order[i] (or i when order is null); item = unit * pairs + pair of
  // 128-row query blocks
  const int* order;
  int pairs;
  // Thread blocks from half_from on take one query block each: block half_from + 2 i + t the t-th of the item that block
  // half_from + i would have.  The launcher cuts the items of a last wave that is less than half full, as the dense kernels'.
  int half_from;
  // optional [BH, nqb]: query blocks with route != 0 are computed by the block-route kernel and are left
  // alone here (no loads, no stores)
  const int* route;
  float scale_log2;
};

template <int D>
struct TokenCfg {
  static constexpr int kHalves = D / 64;
  static constexpr int kTileBytes = 128 * D * 2;
  static constexpr int kStages = (D == 128) ? 4 : 8;
  // Seven gather warps keep up: the copies wait for nothing but free stages (a bare gather of the same rows by eight warps
  // runs at 19 TB/s, three times what this kernel draws).  What bounds a step is the softmax and the round trip through
  // the products, so the registers go to the softmax warps (208), which hold a row's 128 scores and read them from tensor
  // memory once.  With fifteen gather warps the softmax had 152 and read them twice, 32 at a time: 12 heads of 32760 rows,
  // D = 128, 3276 keys of every block 0.896 -> 0.752 ms, threshold lists (1626 on average) 0.474 -> 0.414; D = 64 0.757 ->
  // 0.724 and 0.402 -> 0.378.
  static constexpr int kGatherWarps = 7;
  static constexpr int kGatherThreads = 32 * kGatherWarps;
  static constexpr int kThreads = 32 * (8 + 1 + kGatherWarps);   // 8 softmax warps, the UMMA issuer, the gather warps
  static constexpr int kOffQ = 0;
  static constexpr int kOffRing = 2 * kTileBytes;
  static constexpr int kOffBar = kOffRing + kStages * kTileBytes;
  static constexpr int kSmemBytes = kOffBar + 1024 + 1024;
};

enum : int { TB_Q_FULL = 0, TB_FULL = 1, TB_EMPTY = 9, TB_S_FULL = 17, TB_P_FULL = 19, TB_O_FULL = 21, TB_COUNT = 23 };

__device__ __forceinline__ void cp_async_16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }


template <int D>
__global__ void __launch_bounds__(TokenCfg<D>::kThreads, 1)
sparse_token_attn_kernel(const __grid_constant__ CUtensorMap mq, const __grid_constant__ CUtensorMap mo,
                         const TokenParams p) {
  using Cfg = TokenCfg<D>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const uint32_t sbase = smem_u32(smem);
  const uint32_t bars = sbase + Cfg::kOffBar;
  auto bar = [&](int i) -> uint32_t { return bars + 8u * uint32_t(i); };
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + Cfg::kOffBar + 8 * TB_COUNT);
  AbortState* ab = reinterpret_cast<AbortState*>(smem + Cfg::kOffBar + 8 * TB_COUNT + 8);

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  grid_wait();                                           // for lists and order (launch_behind)
  const int half = int(blockIdx.x) - p.half_from;        // >= 0: one query block of an item
  const int place = half < 0 ? int(blockIdx.x) : p.half_from + (half >> 1);
  const int item = p.order ? p.order[place] : place;
  const int bh = item / p.pairs;
  const int q0 = (item - bh * p.pairs) * 256;
  bool skip[2] = {half >= 0 && (half & 1) != 0, half >= 0 && (half & 1) == 0};
  if (p.route) {
#pragma unroll
    for (int t = 0; t < 2; ++t) {
      const int qb = (q0 >> 7) + t;
      skip[t] |= qb >= p.nqb || p.route[size_t(bh) * p.nqb + qb] != 0;
    }
    if (skip[0] && skip[1]) return;                      // CTA-uniform, before any set-up
  }

  if (tid == 0) {
    ab->flag = 0;
    mbar_init(bar(TB_Q_FULL), 1);
    for (int s = 0; s < 8; ++s) {
      mbar_init(bar(TB_FULL + s), Cfg::kGatherThreads);
      mbar_init(bar(TB_EMPTY + s), 1);
    }
    for (int t = 0; t < 2; ++t) {
      mbar_init(bar(TB_S_FULL + t), 1);
      mbar_init(bar(TB_P_FULL + t), 128);
      mbar_init(bar(TB_O_FULL + t), 1);
    }
    mbar_fence_init();
  }
  if (warp == 8) {
    __syncwarp();
    tmem_alloc(smem_u32(tmem_slot), 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  // per-slot list length and number of 128-token steps; slot t's list starts at lst + t * mask_stride
  auto list_length = [&](int t) {
    const int qb = (q0 >> 7) + t;
    const bool none = qb >= p.nqb || (t ? skip[1] : skip[0]);
    return none ? 0 : max(0, min(p.kv_cnt[size_t(bh) * p.nqb + qb], p.mask_stride));
  };
  const int cnt0 = list_length(0), cnt1 = list_length(1);
  const int* const lst = p.kv_idx + (size_t(bh) * p.nqb + (q0 >> 7)) * p.mask_stride;
  const int nst0 = (cnt0 + 127) >> 7, nst1 = (cnt1 + 127) >> 7, n_max = max(nst0, nst1);

  if (warp == 8 || warp >= 10) {
    // ------------------------------------------------------------------ gather producers
    reg_dealloc<48>();
    if (warp == 8 && lane == 0) {
      tma_prefetch_desc(&mq);
      tma_prefetch_desc(&mo);
      mbar_arrive_expect_tx(bar(TB_Q_FULL), 2 * Cfg::kTileBytes);
      for (int t = 0; t < 2; ++t)
        for (int h = 0; h < Cfg::kHalves; ++h)
          tma_load_3d(sbase + Cfg::kOffQ + t * Cfg::kTileBytes + h * 16384, &mq, bar(TB_Q_FULL), h * 64, q0 + t * 128,
                      bh);
    }
    __syncwarp();
    const int gw = (warp == 8) ? 0 : warp - 9;                         // gather warp 0..6
    constexpr int kChunksPerRow = D / 8;                               // 16-byte chunks per row
    constexpr int kRowsPerInstr = 32 / kChunksPerRow;                  // rows one warp-wide copy covers
    // rows of a 128-token tile are dealt to the seven gather warps in contiguous runs of 4 x 20 + 3 x 16; a lane
    // keeps the token id of run row `lane`
    const int row0 = (gw < 4) ? gw * 20 : 80 + (gw - 4) * 16, nrows = (gw < 4) ? 20 : 16;
    const int sub = lane / kChunksPerRow, ch = lane % kChunksPerRow;
    int idx = 0;
    bool ok = true;
    int pending_stage = -1;                                            // tile whose copies are in flight
    // Token ids of the slots' current steps, and the entries of the steps after them, requested a step ahead: asked for when
    // their tile is next, they held up that tile and the signal of the one before it (3276 keys of 32760, 12 heads, D = 128
    // 0.752 -> 0.710 ms, D = 64 0.724 -> 0.639; threshold lists 0.414 -> 0.405 and 0.378 -> 0.348).  The copies' own
    // asynchronous arrival on the stage barriers instead of the wait for the tile before: level; an UMMA issuer per slot
    // (and six gather warps): 4-13 % slower.
    int tok0 = 0, tok1 = 0, next0 = 0, next1 = 0;
    auto request = [&](int t, int j) {
      const int pos = j * 128 + row0 + lane;
      const int a = (lane < nrows && pos < (t ? cnt1 : cnt0)) ? lst[(t ? p.mask_stride : 0) + pos] : 0;
      if (t) next1 = a;
      else next0 = a;
    };
    auto take_tokens = [&](int t, int j) {                                 // j: the step taken
      const int a = t ? next1 : next0;
      const int tok = (a < 0 || a >= p.S_kv) ? 0 : a;                      // masked column: any finite row will do
      if (t) tok1 = tok;
      else tok0 = tok;
      request(t, j + 1);
    };
    request(0, 0);
    request(1, 0);
    // Each copy instruction moves whole rows: 16 (D = 128) or 8 (D = 64) neighbouring lanes fetch the
    // consecutive 16-byte chunks of one row, so a warp-wide copy asks L2 for full 128-byte lines
    // instead of 32 separate sectors.
    auto gather_tile = [&](const __nv_bfloat16* base, int t) {
      const int st = idx % Cfg::kStages, f = idx / Cfg::kStages;
      if (f > 0) ok = mbar_wait(bar(TB_EMPTY + st), (f - 1) & 1, ab, p.err, 701);
      if (!ok) return;
      const uint32_t dst = sbase + Cfg::kOffRing + st * Cfg::kTileBytes + (ch >> 3) * 16384;
      const __nv_bfloat16* src0 = base + size_t(bh) * p.S_kv * D + ch * 8;
      for (int r = 0; r < nrows; r += kRowsPerInstr) {                 // nrows is a multiple of 4
        const int lr = r + sub;                                        // run row of this lane
        const int tok = __shfl_sync(0xffffffffu, t ? tok1 : tok0, lr);
        cp_async_16(dst + sw128_offset(row0 + lr, ch & 7), src0 + size_t(tok) * D);
      }
      cp_async_commit();
      if (pending_stage >= 0) {
        cp_async_wait<1>();                                            // the previous tile has landed
        fence_proxy_async_smem();
        mbar_arrive(bar(TB_FULL + pending_stage));
      }
      pending_stage = st;
      ++idx;
    };
    // order: K(0,0) K(1,0), then per step V(t,j) K(t,j+1); the ids of step j serve K(t,j) and V(t,j)
    if (nst0 > 0) { take_tokens(0, 0); gather_tile(p.k, 0); }
    if (nst1 > 0 && ok) { take_tokens(1, 0); gather_tile(p.k, 1); }
    for (int j = 0; j < n_max && ok; ++j) {
#pragma unroll
      for (int t = 0; t < 2; ++t) {
        const int n = t ? nst1 : nst0;
        if (ok && j < n) {
          gather_tile(p.v, t);
          if (ok && j + 1 < n) {
            take_tokens(t, j + 1);
            gather_tile(p.k, t);
          }
        }
      }
    }
    cp_async_wait<0>();
    if (ok && pending_stage >= 0) {
      fence_proxy_async_smem();
      mbar_arrive(bar(TB_FULL + pending_stage));
    }
    if (!ok && warp == 8 && lane == 0) mbar_wait_brief(bar(TB_Q_FULL), 0);
  } else if (warp == 9) {
    // ------------------------------------------------------------------ UMMA issuer
    reg_dealloc<48>();
    {   // whole warp, uniform control flow; single instructions go through an elected lane
      const uint32_t idesc_qk = umma_idesc_bf16(128, 128, false);
      const uint32_t idesc_pv = umma_idesc_bf16(128, D, true);
      int idx = 0;
      bool ok = mbar_wait_warp(bar(TB_Q_FULL), 0, ab, p.err, 801);
      auto qk = [&](int t) {
        const int st = idx % Cfg::kStages;
        ok = mbar_wait_warp(bar(TB_FULL + st), (idx / Cfg::kStages) & 1, ab, p.err, 802);
        if (!ok) return;
        tc_fence_after();
        const uint32_t qa = sbase + Cfg::kOffQ + t * Cfg::kTileBytes, ka = sbase + Cfg::kOffRing + st * Cfg::kTileBytes;
        if (elect_one()) {             // one election for the product and its commits
#pragma unroll
          for (int ks = 0; ks < D / 16; ++ks) {
            const uint32_t off = (ks / 4) * 16384 + (ks % 4) * 32;
            umma_ss(tmem + t * 128, umma_smem_desc_sw128(qa + off, 16, 1024), umma_smem_desc_sw128(ka + off, 16, 1024),
                    idesc_qk, ks > 0);
          }
          umma_commit(bar(TB_S_FULL + t));
          umma_commit(bar(TB_EMPTY + st));
        }
        __syncwarp();
        ++idx;
      };
      auto pv = [&](int t, int j) {
        const int st = idx % Cfg::kStages;
        ok = mbar_wait_warp(bar(TB_FULL + st), (idx / Cfg::kStages) & 1, ab, p.err, 803);
        if (ok) ok = mbar_wait_warp(bar(TB_P_FULL + t), j & 1, ab, p.err, 804);
        if (!ok) return;
        tc_fence_after();
        const uint32_t va = sbase + Cfg::kOffRing + st * Cfg::kTileBytes;
        if (elect_one()) {
#pragma unroll
          for (int ks = 0; ks < 8; ++ks)
            umma_ts(tmem + 256 + t * 128, tmem + t * 128 + ks * 8, umma_smem_desc_sw128(va + ks * 2048, 16384, 1024),
                    idesc_pv, (j > 0 || ks > 0) ? 1u : 0u);
          umma_commit(bar(TB_EMPTY + st));
        }
        __syncwarp();
        ++idx;
      };
      // the tiles in the order of the gather warps
      if (ok && nst0 > 0) qk(0);
      if (ok && nst1 > 0) qk(1);
      for (int j = 0; j < n_max && ok; ++j) {
        for (int t = 0; t < 2 && ok; ++t) {
          const int n = t ? nst1 : nst0;
          if (j < n) {
            pv(t, j);
            if (!ok) break;
            if (j + 1 < n) qk(t);
            else umma_commit_elect(bar(TB_O_FULL + t));
          }
        }
      }
    }
  } else {
    // ------------------------------------------------------------------ softmax warpgroups
    reg_alloc<208>();
    const int t = warp >> 2, wq = warp & 3;
    const int row = q0 + t * 128 + wq * 32 + lane;
    const uint32_t lane_base = tmem + (uint32_t(wq * 32) << 16);
    const uint32_t s_addr = lane_base + t * 128, o_addr = lane_base + 256 + t * 128;
    OnlineState st;
    online_init(st);
    bool ok = true;
    // Which of a step's 128 gathered columns are real keys: the entries are requested when the step before has been
    // computed and looked at when the step's scores are there.
    const int n_mine = t ? nst1 : nst0, c_mine = t ? cnt1 : cnt0;
    const int* const l_mine = lst + (t ? p.mask_stride : 0) + lane;
    int ahead[4];
    auto request = [&](int j) {
#pragma unroll
      for (int w = 0; w < 4; ++w) {
        const int pos = j * 128 + w * 32;
        ahead[w] = (pos + lane < c_mine) ? l_mine[pos] : -1;
      }
    };
    request(0);
    for (int j = 0; j < n_mine; ++j) {
      ok = mbar_wait(bar(TB_S_FULL + t), j & 1, ab, p.err, 901);
      if (!ok) break;
      tc_fence_after();
      uint32_t live[4];
#pragma unroll
      for (int w = 0; w < 4; ++w) live[w] = __ballot_sync(0xffffffffu, ahead[w] >= 0 && ahead[w] < p.S_kv);
      float mx0, mx1;
      // full steps start their exponentials before the maximum is known (softmax_steps.cuh): top-k lists 0.720 -> 0.697 ms,
      // threshold lists 0.416 -> 0.399, D = 64 0.642 -> 0.629 and 0.351 -> 0.346, the same bits.  A share of the
      // exponentials on the FMA pipe: level to 5 % slower.
      // Every listed key takes its exponential, however small: NaN and infinities of K and V rows reach the output.  Listed
      // keys are hardly ever negligible for 32 rows, so the test for it cost more than it saved: threshold lists 0.390 ->
      // 0.369 ms, D = 64 0.353 -> 0.337; top-k lists level and 0.642 -> 0.609.
      if (j > 0 && (live[0] & live[1] & live[2] & live[3]) == 0xffffffffu)
        softmax_steady_step<D, 0, false>(s_addr, s_addr, o_addr, p.scale_log2, st, mx0, mx1);
      else
        softmax_online_step<D, true, 0, false>(s_addr, s_addr, o_addr, 64, 64, p.scale_log2, j == 0, st, mx0, mx1, live);
      tc_fence_before();
      mbar_arrive(bar(TB_P_FULL + t));
      request(j + 1);
    }
    __nv_bfloat16* orow = p.o + (size_t(bh) * p.S + row) * D;
    if (t ? skip[1] : skip[0]) {
      // another kernel owns these rows
    } else if (n_mine == 0) {
      if (row < p.S) {
#pragma unroll
        for (int i = 0; i < D / 8; ++i) reinterpret_cast<uint4*>(orow)[i] = make_uint4(0, 0, 0, 0);
      }
    } else if (ok) {
      ok = mbar_wait(bar(TB_O_FULL + t), 0, ab, p.err, 902);
      if (ok) {
        tc_fence_after();
        // the slot's Q tile has been read by its last product: it serves as the output buffer
        store_o_warp<D>(o_addr, sbase + Cfg::kOffQ + t * Cfg::kTileBytes + wq * 4096, &mo, st.l > 0.f ? 1.0f / st.l : 0.f,
                        q0 + t * 128 + wq * 32, bh, q0 + t * 128 + wq * 32 < p.S, lane);
        if (lane == 0) bulk_wait_read();
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 8) {
    __syncwarp();
    tmem_dealloc(tmem, 512);
  }
}

}  // namespace fg
