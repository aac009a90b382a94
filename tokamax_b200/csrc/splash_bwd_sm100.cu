// Splash attention backward for sm_100a: bf16 inputs, head_dim 128, fp32 accumulation.
//
// Two forms.  The split form is atomic-free and bitwise repeatable in all three gradients:
//   1. delta      : -di[b,h,q] = -sum_d o * do  (stored negated: dP + (-di) is an add, which has a
//                   two-wide form)                                   (HBM-bound elementwise pass)
//   2. dq kernel  : one CTA per (q tile, q head).  Per kv tile: S = Q K^T, dP = dO V^T,
//                   dS = P o (dP - di), dQ += dS K.
//   3. dkv kernel : one CTA per (kv tile, kv head).  Loops over the q heads that share the kv
//                   head and their active q tiles: S^T = K Q^T, dP^T = V dO^T, dV += P^T dO,
//                   dK += dS^T Q.  The whole GQA group is summed in the CTA's fp32 TMEM
//                   accumulators, so dK/dV need no atomics and no second pass.
// The fused form (SPLASH_BWD_FUSED_DQ) is what the reference's live backward does — one kernel,
// five matmuls per live block (splash_attention_kernel.py:1234-1459, dq partials :1395-1410
// reduced at :1864): the dkv kernel also forms dQ_partial = dS K for every (q tile, kv tile) pair
// it visits, from the dS^T tile it already holds in shared memory, and adds it into an fp32 dQ
// image in global memory (bulk reductions, sent by eight drain warps); a last HBM-bound pass scales
// and casts that image to bf16.  S and dP are then computed once per pair instead of twice (5
// tile-MMAs instead of 7).  dK / dV stay atomic-free and repeatable; dQ's fp32 sums arrive in an
// order that varies from run to run, so its last bits are not repeatable in this form.
// P (and dS in the dq kernel) is written back to TMEM as bf16 and consumed as the A operand of the
// next MMA; the dkv kernel's dS^T goes through shared memory instead, which frees its TMEM columns
// a step earlier.  K, V, Q and dO tiles are each staged once by TMA and read both K-major and
// MN-major from the same 128-byte-swizzled shared-memory image.
//
// Arithmetic follows the reference backward
// (tokamax/_src/ops/experimental/tpu/splash_attention/splash_attention_kernel.py:1234-1459 and
// base.py:115-173): P = exp(S - logsumexp), dS = (dP - di) * P, with the softmax scale applied
// in fp32 inside the kernels.
#include <mutex>

#include "splash_common.cuh"
#include "splash_bwd_params.cuh"
#include "splash_split.cuh"

namespace sb {

constexpr int kBwdStages = 4;
constexpr int kDqStages = 5;  // K/V ring of the dq kernel: 2.5 steps of look-ahead

// ------------------------------------------------------------------------------------------
// delta = rowsum(o * do)
// ------------------------------------------------------------------------------------------
struct DeltaParams {
  const __nv_bfloat16* o;
  const __nv_bfloat16* d_o;
  int64_t o_sb, o_sh, o_ss, do_sb, do_sh, do_ss;
  float* delta;      // [B, Hq, Sq]  -sum_d(o * do)
  const float* lse;  // [B, Hq, Sq] natural log
  float* nlse2;      // [B, Hq, Sq]  -lse * log2(e): the exponent offset the MMA kernels subtract
  int q_heads, q_len;
  int d_v;  // columns of o / do
  // fused backward: the fp32 dQ image (one 128 x 128 tile per 128 rows, see BwdParams::dq_acc)
  // that the reductions of the dkv kernel add into; this pass clears it on the way.  nullptr: none.
  float* dq_image;
  int dq_chunks;  // 32-column chunks of the image that hold columns of dq
};

// 64 rows per block: a warp takes eight rows, half a warp per row (16 lanes x 16 bytes = one row of
// 128 bf16), four rows deep, with all eight 16-byte loads of a lane in flight before the first is
// used (the pass is a pure stream: 512 bytes read and 8 written per row; with the image 512 more written).
// 32768 rows x 32 (1.09 GB with the image): 0.158 ms = 6.9 TB/s, 1.05 of the measured copy rate; it took 0.245
// while every lane divided its four row numbers by 64-bit lengths and the image was cleared ahead of the loads.
constexpr int kDeltaRowsPerBlock = 64;
__global__ void __launch_bounds__(256) splash_delta_kernel(const DeltaParams p) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int sub = lane & 15, half = lane >> 4;
  // q_len is a multiple of 128, so a block's 64 rows belong to one (batch, head): one division a block
  const int64_t first = (int64_t)blockIdx.x * kDeltaRowsPerBlock;
  const int64_t bh = first / p.q_len;
  const int64_t b = bh / p.q_heads;
  const int h = (int)(bh - b * p.q_heads), q0 = (int)(first - bh * p.q_len) + warp * 8 + half;
  const int64_t row0 = first + warp * 8 + half;
  const __nv_bfloat16* o_base = p.o + b * p.o_sb + h * p.o_sh;
  const __nv_bfloat16* do_base = p.d_o + b * p.do_sb + h * p.do_sh;
  float acc[4] = {0.f, 0.f, 0.f, 0.f};
  // one pass per 128 columns (a second one only for head dims above 128)
  for (int c0 = 0; c0 < p.d_v; c0 += kHeadDim) {
    uint4 a[4], g[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      a[i] = make_uint4(0u, 0u, 0u, 0u);
      g[i] = a[i];
      if (c0 + sub * 8 < p.d_v) {
        a[i] = __ldcs(reinterpret_cast<const uint4*>(o_base + (int64_t)(q0 + 2 * i) * p.o_ss + c0) + sub);
        g[i] = __ldg(reinterpret_cast<const uint4*>(do_base + (int64_t)(q0 + 2 * i) * p.do_ss + c0) + sub);
      }
    }
    if (c0 == 0 && p.dq_image != nullptr) {
      // The block's 64 rows are half of one image tile: in each 32-column chunk a run of 8 KiB.  256 threads x two stores
      // of 16 bytes for each, issued under the loads.
      float* tile = p.dq_image + (first / kTile) * (int64_t)(kTile * kHeadDim) + (first % kTile) * 32;
      const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
      auto clear = [&](int chunk) {
#pragma unroll
        for (int i = 0; i < 2; ++i)
          *reinterpret_cast<uint4*>(tile + chunk * (kTile * 32) + ((i * 256 + (int)threadIdx.x) << 2)) = zero;
      };
      if (p.dq_chunks == 4) {  // (a straight run of stores: tests between them cost this pass a fifth)
#pragma unroll
        for (int chunk = 0; chunk < 4; ++chunk) clear(chunk);
      } else {
        for (int chunk = 0; chunk < p.dq_chunks; ++chunk) clear(chunk);
      }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const uint32_t aw[4] = {a[i].x, a[i].y, a[i].z, a[i].w}, gw[4] = {g[i].x, g[i].y, g[i].z, g[i].w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const __nv_bfloat162 x = *reinterpret_cast<const __nv_bfloat162*>(&aw[j]);
        const __nv_bfloat162 y = *reinterpret_cast<const __nv_bfloat162*>(&gw[j]);
        acc[i] = fmaf(__bfloat162float(x.x), __bfloat162float(y.x), acc[i]);
        acc[i] = fmaf(__bfloat162float(x.y), __bfloat162float(y.y), acc[i]);
      }
    }
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float sum = acc[i];
#pragma unroll
    for (int off = 8; off > 0; off >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, off);
    const int64_t row = row0 + 2 * i;
    if (sub == 0) {
      p.delta[row] = -sum;
      // Rows that never met a live key carry the mask value as logsumexp; -inf keeps their
      // probabilities at exactly zero instead of overflowing the product to +inf.
      const float lse = p.lse[row];
      p.nlse2[row] = lse < -1.0e20f ? -INFINITY : -lse * kLog2e;
    }
  }
}

// ------------------------------------------------------------------------------------------
// shared pieces of the two MMA kernels
// ------------------------------------------------------------------------------------------
constexpr uint32_t kBwdWork = 2;

struct BwdBarriers {
  uint64_t answer[2];  // cluster launch control: what the request for the next tile returned
  // tiles in the order they are worked on: q tile (-1: none left), (batch, q head), first and last entry
  int4 work[kBwdWork];
  uint64_t answer_full;
  uint64_t work_full[kBwdWork], work_empty[kBwdWork];
  uint64_t out_free;                  // a tile's dQ has been read from TMEM (8 arrivals)
  uint64_t stat_full[2];              // stationary operand tiles
  uint64_t ring_full[kDqStages];
  uint64_t ring_empty[kDqStages];
  uint64_t s_full[2];
  uint64_t dp_full;
  uint64_t ds_full;
  uint64_t acc_done;
  uint32_t tmem_base;
  uint32_t abort_flag;
  uint32_t early_exit;
};

constexpr int kDqSmemBytes = (2 + kDqStages) * kTileBytes + 1024 + 1024;

// ------------------------------------------------------------------------------------------
// dq kernel
// ------------------------------------------------------------------------------------------
// TMEM: S0 [0,128) | S1 [128,256) | dP [256,384) | dQ [384,512)
// CTAs stay for several tiles, as the dkv kernel's do: a whole pass of causal 2 x 4096, 16 / 1 heads
// takes 497 -> 493 us at d 64, 576 -> 566 at d 128; 4 x 4096, 16 / 8: 1107 -> 1089.
template <bool kSoftCap>
__global__ void __launch_bounds__(kBwdThreads, 1)
splash_dq_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_do,
                 const __grid_constant__ CUtensorMap tm_k, const __grid_constant__ CUtensorMap tm_v,
                 const BwdParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  uint8_t* q_smem = smem;
  uint8_t* do_smem = smem + kTileBytes;
  uint8_t* ring = smem + 2 * kTileBytes;
  BwdBarriers* bars = reinterpret_cast<BwdBarriers*>(smem + (2 + kDqStages) * kTileBytes);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  // q tile, (batch, q head), first and last entry of a block of the grid
  auto tile_of = [&](unsigned block) {
    const CtaWork t = cta_work_at(block, p.row_order, p.n_rows, p.n_groups, p.chunk_groups, true);
    const int beg = p.row_ptr[t.row];
    const int end = p.row_end ? p.row_end[(int64_t)(t.group / p.q_heads) * p.n_rows + t.row] : p.row_ptr[t.row + 1];
    return make_int4(t.row, t.group, beg, end < beg ? beg : end);
  };
  auto list_of = [&](const int4& w) { return p.entries + (int64_t)(w.y / p.q_heads) * p.entries_per_batch; };

  if (threadIdx.x == 0) {
    bars->early_exit = *reinterpret_cast<volatile uint32_t*>(p.err);
    bars->abort_flag = 0;
    mbar_init(&bars->stat_full[0], 1);
    mbar_init(&bars->stat_full[1], 1);
    for (int s = 0; s < kDqStages; ++s) {
      mbar_init(&bars->ring_full[s], 1);
      mbar_init(&bars->ring_empty[s], 1);
    }
    mbar_init(&bars->s_full[0], 1);
    mbar_init(&bars->s_full[1], 1);
    mbar_init(&bars->dp_full, 1);
    for (uint32_t i = 0; i < kBwdWork; ++i) {
      mbar_init(&bars->work_full[i], 1);
      mbar_init(&bars->work_empty[i], 9);  // compute warps and the issuing one
    }
    mbar_init(&bars->answer_full, 1);
    mbar_init(&bars->out_free, 8);
    mbar_init(&bars->ds_full, 8);  // one arrival per compute warp
    mbar_init(&bars->acc_done, 1);
    mbar_fence_init();
  }
  __syncthreads();
  if (bars->early_exit != 0) return;
  int4 own = make_int4(0, 0, 0, 0);
  if (warp == 8) {  // looked up beside the allocation; the others hear of it from the queue
    own = tile_of(blockIdx.x);
    if (lane == 0) {
      tma_prefetch_desc(&tm_q);
      tma_prefetch_desc(&tm_do);
      tma_prefetch_desc(&tm_k);
      tma_prefetch_desc(&tm_v);
    }
  }
  if (warp == 9) {
    tmem_alloc(&bars->tmem_base, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = bars->tmem_base;
  AbortCtx ab{&bars->abort_flag, p.err};

  // The tiles this CTA works on, in order: its own, then those it takes over (the producer posts both).
  uint32_t taken = 0;  // tiles so far: slot and phase of the next one
  auto work_slot = [&]() { return taken % kBwdWork; };
  auto work_phase = [&]() { return (taken / kBwdWork) & 1u; };
  // Calls body(tile) for each, until it returns false: by a whole warp, or by a thread for its warp.
  auto each_tile = [&](bool warp_wide, auto body) {
    for (;;) {
      bool ok = mbar_wait(&bars->work_full[work_slot()], work_phase(), ab, 0x1700u + work_slot());
      if (warp_wide) ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      const int4 w = bars->work[work_slot()];
      if (w.x < 0) break;
      if (warp_wide) __syncwarp();
      if (!warp_wide || lane == 0) mbar_arrive(&bars->work_empty[work_slot()]);
      ++taken;
      if (!body(w)) break;
    }
  };

  if (warp >= 8) {
   setmaxnreg_dec<kIssueRegs>();
   if (warp == 8) {
    if (elect_one()) {
      // tiles are two 64-column halves; with at most 64 real columns the second is never read
      const bool qk2 = p.d_qk > 64, v2 = p.d_v > 64;
      uint32_t it = 0;
      uint32_t stepped = 0;  // tiles with steps so far
      uint32_t asked = 0;
      bool ok = true;
      int4 w = own;
      while (ok) {
        ok = mbar_wait(&bars->work_empty[work_slot()], work_phase() ^ 1u, ab, 0x1710u + work_slot());
        if (!ok) break;
        bars->work[work_slot()] = w;
        mbar_arrive(&bars->work_full[work_slot()]);
        ++taken;
        if (w.x < 0) break;
        const int4* entries = list_of(w);
        const int head = w.y % p.q_heads, batch = w.y / p.q_heads, kv_head = head / (p.q_heads / p.kv_heads);
        for (int e = w.z; e < w.w && ok; ++e) {
          const int col = entries[e].x;
          for (int kv = 0; kv < 2 && ok; ++kv, ++it) {
            const uint32_t s = it % kDqStages;
            ok = mbar_wait(&bars->ring_empty[s], ((it / kDqStages) & 1u) ^ 1u, ab, 0x1100u + s);
            if (!ok) break;
            uint8_t* dst = ring + s * kTileBytes;
            const CUtensorMap* tm = kv == 0 ? &tm_k : &tm_v;
            const bool two = kv == 0 ? qk2 : v2;
            mbar_arrive_expect_tx(&bars->ring_full[s], two ? kTileBytes : kHalfBytes);
            tma_load_4d(dst, tm, &bars->ring_full[s], 0, col * kTile, kv_head, batch);
            if (two) tma_load_4d(dst + kHalfBytes, tm, &bars->ring_full[s], 64, col * kTile, kv_head, batch);
            if (kv == 0 && e == w.z) {  // Q and dO of the tile, once the MMAs of the last one have read theirs
              if (stepped > 0) ok = mbar_wait(&bars->acc_done, (stepped - 1) & 1u, ab, 0x1120u);
              if (!ok) break;
              mbar_arrive_expect_tx(&bars->stat_full[0], qk2 ? kTileBytes : kHalfBytes);
              tma_load_4d(q_smem, &tm_q, &bars->stat_full[0], 0, w.x * kTile, head, batch);
              if (qk2) tma_load_4d(q_smem + kHalfBytes, &tm_q, &bars->stat_full[0], 64, w.x * kTile, head, batch);
              mbar_arrive_expect_tx(&bars->stat_full[1], v2 ? kTileBytes : kHalfBytes);
              tma_load_4d(do_smem, &tm_do, &bars->stat_full[1], 0, w.x * kTile, head, batch);
              if (v2) tma_load_4d(do_smem + kHalfBytes, &tm_do, &bars->stat_full[1], 64, w.x * kTile, head, batch);
              ++stepped;
            }
          }
        }
        if (!ok) break;
        // The next tile.  Asked for when all of this one is on its way, and no earlier: what a CTA has taken over, no other
        // can take that is done before it.
        mbar_arrive_expect_tx(&bars->answer_full, 16);
        clc_request(bars->answer, &bars->answer_full);
        ok = mbar_wait(&bars->answer_full, asked & 1u, ab, 0x1720u);
        ++asked;
        const int block = ok ? clc_block(bars->answer) : -1;
        fence_proxy_async_smem();  // read before the next answer overwrites it
        w = block >= 0 ? tile_of((unsigned)block) : make_int4(-1, 0, 0, 0);
      }
    }
  } else if (warp == 9) {
    if (elect_one()) {
      constexpr uint32_t idesc_kk = make_idesc_bf16(kTile, kTile, false, false);
      // N of dQ += dS K: dq's columns — 128, or 64 when q / k have at most 64
      const uint32_t idesc_mn = make_idesc_bf16(kTile, p.d_qk <= 64 ? 64 : kHeadDim, false, true);
      const uint32_t q_addr = smem_u32(q_smem), do_addr = smem_u32(do_smem), ring_addr = smem_u32(ring);
      const uint32_t t_dp = tmem + 2 * kTile, t_dq = tmem + 3 * kTile;
      auto ss_kmajor = [&](uint32_t d, uint32_t a0, uint32_t b0, int nk) {
        const SmemDesc da = make_smem_desc_sw128(a0, 16, 1024), db = make_smem_desc_sw128(b0, 16, 1024);
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          if (nk != 8 && k >= nk) break;  // head dims below 128: the remaining slices multiply zeros
          const uint32_t off = (k >> 2) * kHalfBytes + (k & 3) * 32;
          umma_ss(d, desc_at(da, off), desc_at(db, off), idesc_kk, k > 0 ? 1u : 0u);
        }
      };
      auto ring_wait = [&](uint32_t it, uint32_t tag) {
        return mbar_wait(&bars->ring_full[it % kDqStages], (it / kDqStages) & 1u, ab, tag);
      };
      uint32_t n = 0;      // steps so far
      uint32_t tiles = 0;  // tiles with steps so far
      each_tile(false, [&](const int4& w) {
      const uint32_t first = n, last = n + (uint32_t)(w.w - w.z);
      if (first == last) return true;
      // S and dP of the first step
      bool ok = mbar_wait(&bars->stat_full[0], tiles & 1u, ab, 0x1200u) && ring_wait(2 * n, 0x1210u);
      if (ok) {
        mma_issue_fence();
        ss_kmajor(tmem + (n & 1u) * kTile, q_addr, ring_addr + (2 * n % kDqStages) * kTileBytes, p.nk_qk);
        tc_commit(&bars->s_full[n & 1u]);
      }
      ok = ok && mbar_wait(&bars->stat_full[1], tiles & 1u, ab, 0x1201u) && ring_wait(2 * n + 1, 0x1211u);
      if (ok) {
        mma_issue_fence();
        ss_kmajor(t_dp, do_addr, ring_addr + ((2 * n + 1) % kDqStages) * kTileBytes, p.nk_v);
        tc_commit(&bars->dp_full);
        tc_commit(&bars->ring_empty[(2 * n + 1) % kDqStages]);
      }
      // the output of the tile before has been read
      if (tiles > 0) ok = ok && mbar_wait(&bars->out_free, (tiles - 1) & 1u, ab, 0x1260u);
      ++tiles;
      for (; n < last && ok; ++n) {
        const bool has_next = n + 1 < last;
        const uint32_t it_k = 2 * n, it_kn = 2 * n + 2, it_vn = 2 * n + 3;
        if (has_next) {
          ok = ring_wait(it_kn, 0x1220u);
          if (!ok) break;
          mma_issue_fence();
          ss_kmajor(tmem + ((n + 1) & 1) * kTile, q_addr, ring_addr + (it_kn % kDqStages) * kTileBytes, p.nk_qk);
          tc_commit(&bars->s_full[(n + 1) & 1]);
        }
        ok = mbar_wait(&bars->ds_full, n & 1u, ab, 0x1230u);
        if (!ok) break;
        mma_issue_fence();
        {
          // dQ += dS_n K_n : A = packed dS in the S buffer, B = K tile read MN-major.
          const uint32_t a_base = tmem + (n & 1) * kTile;
          const SmemDesc db = make_smem_desc_sw128(ring_addr + (it_k % kDqStages) * kTileBytes, kHalfBytes, 1024);
#pragma unroll
          for (int k = 0; k < 8; ++k)
            umma_ts(t_dq, a_base + packed_a_col(k), desc_at(db, k * 2048), idesc_mn, (n > first || k > 0) ? 1u : 0u);
          tc_commit(&bars->ring_empty[it_k % kDqStages]);
        }
        if (has_next) {
          ok = ring_wait(it_vn, 0x1240u);
          if (!ok) break;
          mma_issue_fence();
          ss_kmajor(t_dp, do_addr, ring_addr + (it_vn % kDqStages) * kTileBytes, p.nk_v);
          tc_commit(&bars->dp_full);
          tc_commit(&bars->ring_empty[it_vn % kDqStages]);
        }
      }
      tc_commit(&bars->acc_done);
      return ok;
      });
    }
   }
  } else {
    // ------------------------------------------------------------------ compute warpgroups
    setmaxnreg_inc<kComputeRegs>();
    const int w = warp >> 2;       // column half this warpgroup owns
    const int wq = warp & 3;
    const int r = wq * 32 + lane;  // q row within the tile
    const bool has_seg = p.q_seg != nullptr;
    const uint32_t lane_addr = (uint32_t)(wq * 32) << 16;
    const float c = kSoftCap ? p.soft_cap * kLog2e : p.scale_log2;
    uint32_t n = 0;      // steps so far
    uint32_t tiles = 0;  // tiles with steps so far
    each_tile(true, [&](const int4& work) {
    const int head = work.y % p.q_heads, batch = work.y / p.q_heads;
    const int4* entries = list_of(work);
    const int n_ent = work.w - work.z;
    const int q_row = work.x * kTile + r;
    const int qi = p.q_sequence ? p.q_sequence[q_row] : q_row;
    const RowInterval iv = mask_fn_interval(p.fn, qi);
    const int q_seg = has_seg ? p.q_seg[(int64_t)batch * p.q_len + q_row] : 0;
    const int32_t* kv_seg_row = has_seg ? p.kv_seg + (int64_t)batch * p.kv_len : nullptr;
    const int64_t stat = ((int64_t)batch * p.q_heads + head) * p.q_len + q_row;
    const float nlse2 = p.nlse2[stat];
    const float ndelta = p.delta[stat];  // -di
    bool ok = true;

    int4 ent_next = n_ent > 0 ? entries[work.z] : make_int4(0, 0, 0, 0);
    for (int e = work.z; e < work.w; ++e, ++n) {
      const int4 ent = ent_next;
      if (e + 1 < work.w) ent_next = entries[e + 1];  // fetched a step ahead of its use
      const int st = ent.y & 3;
      const int kv0 = ent.x * kTile + w * 64;
      const uint32_t t_s = tmem + lane_addr + (n & 1) * kTile;
      ok = mbar_wait(&bars->s_full[n & 1], (n >> 1) & 1u, ab, 0x1400u);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tc_fence_after();
      float pr[64];
      {
        uint32_t v0[32], v1[32];
        tmem_ld32(t_s + w * 64, v0);
        tmem_ld32(t_s + w * 64 + 32, v1);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 32; ++j) {
          pr[j] = __uint_as_float(v0[j]);
          pr[32 + j] = __uint_as_float(v1[j]);
        }
      }
      if constexpr (kSoftCap) {  // pr <- tanh(scale * s / cap), capped before it is masked
        tanh_all(pr, p.softcap_a);
      }
      if (st == 1) {
        if (p.fn.kind != SPLASH_MASK_TABLE) {
          const int lo_rel = iv.lo <= kv0 ? 0 : iv.lo - kv0;
          const int hi_rel = iv.hi >= kv0 + 63 ? 63 : iv.hi - kv0;
#pragma unroll
          for (int j = 0; j < 64; ++j)
            if (j < lo_rel || j > hi_rel) pr[j] = kMaskedLogit;
        } else {
          const int8_t* mrow = p.pmb + ((int64_t)ent.z * p.pm_bq + (q_row % p.pm_bq)) * p.pm_bkv +
                               (kv0 % p.pm_bkv);
          const int4* m4 = reinterpret_cast<const int4*>(mrow);
#pragma unroll
          for (int g = 0; g < 4; ++g) {
            const int4 mv = __ldg(m4 + g);
            const uint32_t wd[4] = {(uint32_t)mv.x, (uint32_t)mv.y, (uint32_t)mv.z, (uint32_t)mv.w};
#pragma unroll
            for (int j = 0; j < 16; ++j)
              if (((wd[j >> 2] >> ((j & 3) * 8)) & 0xffu) == 0u) pr[g * 16 + j] = kMaskedLogit;
          }
        }
      }
      if (has_seg && !((ent.y >> 4) & 1)) {  // (bit set: the whole tile lies inside one segment)
        const int4* sg4 = reinterpret_cast<const int4*>(kv_seg_row + kv0);
#pragma unroll
        for (int g = 0; g < 16; ++g) {
          const int4 sv = __ldg(sg4 + g);
          if (sv.x != q_seg) pr[g * 4 + 0] = kMaskedLogit;
          if (sv.y != q_seg) pr[g * 4 + 1] = kMaskedLogit;
          if (sv.z != q_seg) pr[g * 4 + 2] = kMaskedLogit;
          if (sv.w != q_seg) pr[g * 4 + 3] = kMaskedLogit;
        }
      }
      if constexpr (kSoftCap) {
        // p * (1 - tanh^2): the chain factor of the cap rides on p (masked entries hold -1e30
        // in place of tanh; the clamp keeps their factor finite, their p is 0)
#pragma unroll
        for (int j = 0; j < 64; ++j) {
          const float t = fmaxf(pr[j], -1.0f);
          pr[j] = ex2(fmaf(pr[j], c, nlse2)) * fmaf(-t, t, 1.0f);
        }
      } else {
        // issue-bound: two-wide fp32 fma for the exponent arguments
        const float2 c2 = make_float2(c, c), nl2 = make_float2(nlse2, nlse2);
#pragma unroll
        for (int j = 0; j < 64; j += 2) {
          const float2 x = __ffma2_rn(make_float2(pr[j], pr[j + 1]), c2, nl2);
          pr[j] = ex2(x.x);
          pr[j + 1] = ex2(x.y);
        }
      }

      ok = mbar_wait(&bars->dp_full, n & 1u, ab, 0x1410u);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tc_fence_after();
      uint32_t pk[32];
      {
        uint32_t v0[32], v1[32];
        tmem_ld32(tmem + lane_addr + 2 * kTile + w * 64, v0);
        tmem_ld32(tmem + lane_addr + 2 * kTile + w * 64 + 32, v1);
        tmem_ld_wait();
        const float2 nd2 = make_float2(ndelta, ndelta);
#pragma unroll
        for (int j = 0; j < 16; ++j) {  // dS = p * (dP - di), two elements per instruction
          const float2 a = __fmul2_rn(make_float2(pr[2 * j], pr[2 * j + 1]),
                                      __fadd2_rn(make_float2(__uint_as_float(v0[2 * j]), __uint_as_float(v0[2 * j + 1])), nd2));
          const float2 b = __fmul2_rn(make_float2(pr[32 + 2 * j], pr[32 + 2 * j + 1]),
                                      __fadd2_rn(make_float2(__uint_as_float(v1[2 * j]), __uint_as_float(v1[2 * j + 1])), nd2));
          pk[j] = pack_bf16(a.x, a.y);
          pk[16 + j] = pack_bf16(b.x, b.y);
        }
      }
      tmem_st32(t_s + packed_col(w), pk);
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bars->ds_full);
    }

    // epilogue
    __nv_bfloat16* row0 = p.out0 + (int64_t)batch * p.out0_sb + (int64_t)head * p.out0_sh + (int64_t)(q_row - lane) * p.out0_ss;
    if (n_ent > 0) {
      if (ok) {
        ok = mbar_wait(&bars->acc_done, tiles++ & 1u, ab, 0x1500u);
        ok = __all_sync(0xffffffffu, ok);
      }
      if (ok) {
        tc_fence_after();
#pragma unroll
        for (int g = 0; g < 2; ++g) {
          uint32_t v[32];
          tmem_ld32(tmem + lane_addr + 3 * kTile + w * 64 + g * 32, v);
          tmem_ld_wait();
          if (g == 1) {
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&bars->out_free);
          }
          store_rows32(row0, p.out0_ss, v, p.scale, w * 64 + g * 32, p.d_qk);
        }
      }
    } else {
      uint32_t v[32];
#pragma unroll
      for (int j = 0; j < 32; ++j) v[j] = 0u;
      store_rows32(row0, p.out0_ss, v, 0.f, w * 64, p.d_qk);
      store_rows32(row0, p.out0_ss, v, 0.f, w * 64 + 32, p.d_qk);
    }
    return ok;
    });
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 9) {
    __syncwarp();
    drain_after_give_up(&bars->abort_flag);
    tmem_dealloc(tmem, 512);
  }
}

// ------------------------------------------------------------------------------------------
// dkv kernel
// ------------------------------------------------------------------------------------------
// 16 compute warps (32 kv rows x one 32-column quarter of the q tile each) keep the P^T / dS^T
// phases short; warp 16 feeds TMA, warp 17 issues MMAs, warps 18-19 are idle (they complete the
// fifth warpgroup).
constexpr int kDkvThreads = 640;
constexpr int kDkvTmaWarp = 16;
constexpr int kDkvMmaWarp = 17;
// Fused form: warps 20-27 drain the per-pair dQ tile from TMEM, each 32 lanes of 64 columns: half of that goes through
// 4 KiB of shared memory at once, the other half waits in registers until those have been read, so that the TMEM columns
// are free for the next step's dP^T after two loads.  The image is added to by bulk reductions: an SM sends
// 25 bytes a cycle whichever way (64 KiB a step: 2570 cycles; 3100 beside the step's loads), but vector reds from
// registers, which four warps issued before, stand in the queue that every mbarrier and shared-memory access of the SM goes
// through (the issuing thread saw a finished barrier 1400 cycles late).  4 x 8192, 32 / 8 heads: 5500 -> 4600 cycles a
// step of a CTA in mid-grid, whole pass 7.63 -> 7.35 ms; 8 x 16384, 16 heads, window 4096: 6.99 -> 6.68.  The staging
// takes the slot that a second dO tile had: dO(n) is last read by dV(n), two thousand cycles before dP^T(n + 1) wants the
// next one.  896 threads start at 72 registers.  Registers live in four banks, one per scheduler, and warp w draws on bank
// w mod 4, so every bank serves four compute warps, one warp of the issuing warpgroup and two drain warps: 7 x 72 at
// launch, 4 x 88 + 56 + 2 x 48 after the hand-over (the sum per bank has to stay at what the launch gave it, or the
// increase never completes).
constexpr int kFusedThreads = 896;
constexpr int kDkvDrainWarp = 20;  // the first of
constexpr int kDkvDrainWarps = kFusedThreads / 32 - kDkvDrainWarp;
constexpr int kFusedComputeRegs = 88;
constexpr int kFusedIssueRegs = 56;
constexpr int kFusedDrainRegs = 48;
constexpr int kDqBlockBytes = 32 * 32 * 4;  // a drain warp's share of 32 columns
constexpr int kDqTileFloats = kTile * kHeadDim;
// No register hand-over here: at 640 threads every thread gets 96 registers, which the compute
// warps fit in, and the MMA / TMA threads keep their loop state in registers instead of spilling
// it (with 56 registers the issue loop reloaded descriptor bases from local memory).

// One CTA = one kv tile of one (batch, kv head); the q heads of the GQA group and the active q
// tiles are looped inside and dK / dV of the whole group accumulate in TMEM in fp32 (no atomics,
// bitwise repeatable).  A q tile is processed whole: the score MMAs run with N = 128 (an N = 64 SS
// MMA reads 6 KB of shared memory for 32 cycles of tensor time and so runs at about 60 % of the
// N = 128 rate; a version that double-buffered 64-column halves of the q tile was 21 % slower).
//   TMEM: S^T [0,128) | dP^T [128,256) | dK [256,384) | dV [384,512)
// S^T and dP^T are single-buffered.  P^T goes back to TMEM over S^T (A operand of dV += P^T dO);
// dS^T goes to shared memory in the K-major 128-byte-swizzled layout of an operand tile (A operand
// of dK += dS^T Q), which frees the dP^T columns for the next step as soon as they have been
// read.  Issue order of step n:  wait P^T(n) | dV(n) | S^T(n+1) | wait dS^T(n) | dK(n) | dP^T(n+1)
// (fused: dQ_partial(n) ahead of dK(n), and in most cases S^T(n+1) between the two) — the tensor pipe executes in order, so S^T(n+1) cannot overtake dV(n)'s read of P^T(n), and
// dP^T(n+1) is issued only after the compute warps have consumed dP^T(n).
constexpr int kDkvStatsBytes = (kBwdStages / 2) * 2 * kTile * 4;
constexpr int kDkvSmemBytes = (3 + kBwdStages) * kTileBytes + kDkvStatsBytes + 512;

constexpr uint32_t kDkvWork = 2;

struct DkvBarriers {
  uint64_t answer[2];  // cluster launch control: what the request for the next tile returned
  // tiles in the order they are worked on: kv tile (-1: none left), (batch, kv head), first and last entry
  int4 work[kDkvWork];
  uint64_t answer_full;
  uint64_t work_full[kDkvWork], work_empty[kDkvWork];
  uint64_t out_free;  // a tile's dK and dV have been read from TMEM (16 arrivals)
  uint64_t stat_full[2];
  uint64_t ring_full[kBwdStages];
  uint64_t ring_empty[kBwdStages];
  uint64_t st_full;
  uint64_t dpt_full;
  uint64_t p_full;
  uint64_t ds_full;
  uint64_t ds_free;   // dK(n) has finished reading the dS^T tile in shared memory
  uint64_t acc_done;
  uint64_t dq_full;   // fused: dQ_partial(n) is complete in the dP^T columns
  uint64_t dq_free;   // fused: the drain warps have read it out (kDkvDrainWarps arrivals)
  uint32_t tmem_base;
  uint32_t abort_flag;
  uint32_t early_exit;
  uint32_t n_steps;   // kSplit: steps of this CTA
  int4 step[kBwdStages / 2];  // kSplit: schedule entries of the steps in the ring, covered by their Q slots' barriers
};
static_assert(sizeof(DkvBarriers) <= 512, "barrier block");

// kLateS (fused form): S^T(n+1) is issued behind dQ(n).  Right behind dV(n) it takes all of the shared memory's rate from
// the compute warps, which read dP^T's statistics and write dS^T then; behind dQ(n) it runs under the drain.  late_scores() has
// the rule.
//
// CTAs stay for several tiles: the producer takes over CTAs that have not been launched yet (cluster launch control) when all
// loads of its tile are on their way, posts their tiles and goes on loading; the next tile's first scores are computed while
// the compute warps store dK and dV.  A tile a CTA spent about 20000 cycles between its last step and its successor's
// first.  One tile a CTA -> this, us a pass: 8 x 16384, 16 heads, window 4096 and documents (some 12 steps a tile) 6584 -> 6260,
// causal 4 x 2048, 16 / 16 359 -> 334, 4 x 8192, 32 / 8 6974 -> 6842, prefix 2 x 4096, 16 / 4 617 -> 597 (with the drain
// below, 604 before).  With a soft cap, whole backward: 156 tiles (3 x 1664, 12 / 4 heads, d 80, window 768)
// 91.0 -> 89.2, 248 (causal 3968, 32 / 8) 368 -> 368, 256 (causal 2 x 4096, 16 / 4) 378 -> 382, 260 (5 x 1664, 12 / 4, d 80, window
// 768) 145 -> 141, 1024 (causal 4 x 4096, 16 / 8) 756 -> 738.
//
// kSplit: a cluster of 2 .. 8 CTAs shares one kv tile, each taking its part of the steps (q head, q tile), see PartWalk.
// At the end every CTA leaves its dK and dV (fp32) in its own shared memory and the cluster adds them
// up over distributed shared memory in rank order, each CTA a share of the columns: no atomics, still
// bitwise repeatable.  For grids that leave SMs idle; split_for() holds the rule.
constexpr int kDkvPartWords = 2 * kHeadDim / 4 * kTile;  // 16-byte words: [dk, dv column / 4][kv row]
static_assert(kDkvPartWords * 16 <= (3 + kBwdStages) * kTileBytes, "the parts lie over the operand tiles");

template <bool kSoftCap, bool kFuseDq, bool kSplit, bool kLateS>
__global__ void __launch_bounds__(kFuseDq ? kFusedThreads : kDkvThreads, 1)
splash_dkv_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_do,
                       const __grid_constant__ CUtensorMap tm_k, const __grid_constant__ CUtensorMap tm_v,
                       const BwdParams p) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = smem_raw;
  uint8_t* k_smem = smem;
  uint8_t* v_smem = smem + kTileBytes;
  uint8_t* ds_smem = smem + 2 * kTileBytes;
  uint8_t* ring = smem + 3 * kTileBytes;
  float* stats = reinterpret_cast<float*>(smem + (3 + kBwdStages) * kTileBytes);
  DkvBarriers* bars = reinterpret_cast<DkvBarriers*>(smem + (3 + kBwdStages) * kTileBytes + kDkvStatsBytes);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const unsigned rank = kSplit ? cluster_rank() : 0u;
  const int group = p.q_heads / p.kv_heads;
  // kv tile, (batch, kv head), first and last entry of a block of the grid
  auto tile_of = [&](unsigned block) {
    const unsigned main = (unsigned)(p.main_groups * p.n_rows);
    CtaWork t;
    if (block < main) {
      t = cta_work_at(block, p.row_order, p.n_rows, p.main_groups, p.chunk_groups, false);
    } else {
      const int rest = p.n_groups - p.main_groups;
      t = cta_work_at(block - main, p.row_order, p.n_rows, rest, rest, false);
      t.group += p.main_groups;
    }
    const int beg = p.row_ptr[t.row];
    const int end = p.row_end ? p.row_end[(int64_t)(t.group / p.kv_heads) * p.n_rows + t.row] : p.row_ptr[t.row + 1];
    return make_int4(t.row, t.group, beg, end < beg ? beg : end);
  };
  auto list_of = [&](const int4& w) { return p.entries + (int64_t)(w.y / p.kv_heads) * p.entries_per_batch; };
  // Q and dO of step n in the ring: slots 0, 2 and 1, 3 by turns.  The fused form parks dQ in slot 3: dO then keeps to
  // slot 1, whose two halves take turns where dO has one half.
  const bool one_do = kFuseDq && p.d_v > 64;
  auto do_bar = [&](uint32_t n) { return one_do ? 1u : 1u + 2u * (n & 1u); };
  auto do_phase = [&](uint32_t n) { return (one_do ? n : n >> 1) & 1u; };
  auto do_offset = [&](uint32_t n) { return kTileBytes + (one_do ? 0u : (n & 1u) * (kFuseDq ? kHalfBytes : 2 * kTileBytes)); };
  // steps of a tile: (q head g of the group, entry e) pairs in that order; `offset` (kSplit): of head g's part, a tile less
  // for each further head
  int4 own = kSplit ? tile_of(blockIdx.x / p.n_split) : make_int4(0, 0, 0, 0);
  auto walk_of = [&](const int4& w) { return PartWalk<kSplit>(list_of(w), w.z, w.w, p.n_split); };
  auto offset_behind = [&](int offset) { return kSplit ? (offset == 0 ? p.n_split : offset) - 1 : 0; };

  if (threadIdx.x == 0) {
    // The operand tiles need a 1024-byte aligned base for the 128-byte swizzle; there is no
    // slack in the allocation to fix it up, so a misaligned window is reported, not used.
    uint32_t bad = *reinterpret_cast<volatile uint32_t*>(p.err);
    if ((smem_u32(smem) & 1023u) != 0u) {
      if (atomicCAS(p.err, 0u, 2u) == 0u) {
        p.err[1] = blockIdx.x;
        p.err[2] = 0x2f00u;
        p.err[3] = smem_u32(smem);
      }
      bad = 2u;
    }
    bars->early_exit = bad;
    bars->abort_flag = kSplit ? bad : 0u;  // (read by the other CTAs of the cluster)
    bars->n_steps = 0;
    for (uint32_t i = 0; i < kDkvWork; ++i) {
      mbar_init(&bars->work_full[i], 1);
      mbar_init(&bars->work_empty[i], 17 + (kFuseDq ? kDkvDrainWarps : 0));  // compute, MMA, drain warps
    }
    mbar_init(&bars->answer_full, 1);
    mbar_init(&bars->out_free, 16);
    mbar_init(&bars->stat_full[0], 1);
    mbar_init(&bars->stat_full[1], 1);
    for (int s = 0; s < kBwdStages; ++s) {
      mbar_init(&bars->ring_full[s], 1);
      mbar_init(&bars->ring_empty[s], 1);
    }
    mbar_init(&bars->st_full, 1);
    mbar_init(&bars->dpt_full, 1);
    mbar_init(&bars->p_full, 16);   // one arrival per compute warp
    mbar_init(&bars->ds_full, 16);
    mbar_init(&bars->ds_free, 1);
    mbar_init(&bars->acc_done, 1);
    mbar_init(&bars->dq_full, 1);
    mbar_init(&bars->dq_free, kDkvDrainWarps);
    mbar_fence_init();
  }
  __syncthreads();
  if (bars->early_exit != 0) {
    if constexpr (kSplit) {  // the others may not have seen it: no CTA leaves while its shared memory may be read
      cluster_sync();
      cluster_sync();
    }
    return;
  }
  if constexpr (kSplit) {
    const PartWalk<kSplit> walk = walk_of(own);
    unsigned mine = 0;
    for (int e = own.z + (int)threadIdx.x; e < own.w; e += (int)blockDim.x) {
      const int part = (list_of(own)[e].x - walk.first_tile) % p.n_split;
      for (int g = 0, o = walk.offset((int)rank); g < group; ++g, o = offset_behind(o)) mine += part == o;
    }
    mine = __reduce_add_sync(0xffffffffu, mine);
    if (lane == 0) atomicAdd(&bars->n_steps, mine);
  }
  if (!kSplit && warp == kDkvTmaWarp) {  // looked up beside the allocation; the others hear of it from the queue
    own = tile_of(blockIdx.x);
    if (lane == 0) {
      tma_prefetch_desc(&tm_q);
      tma_prefetch_desc(&tm_do);
      tma_prefetch_desc(&tm_k);
      tma_prefetch_desc(&tm_v);
    }
  }
  if (warp == kDkvMmaWarp) {
    tmem_alloc(&bars->tmem_base, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = bars->tmem_base;
  AbortCtx ab{&bars->abort_flag, p.err};
  auto steps_of = [&](const int4& w) { return kSplit ? bars->n_steps : (uint32_t)((w.w - w.z) * group); };

  // The tiles this CTA works on, in order: its own, then those it takes over (the producer posts both).  kSplit: its own.
  uint32_t taken = 0;  // tiles so far: slot and phase of the next one
  auto work_slot = [&]() { return taken % kDkvWork; };
  auto work_phase = [&]() { return (taken / kDkvWork) & 1u; };
  // Calls body(tile) for each, until it returns false: by a whole warp, or by a thread for its warp.  `hold`: the tile's
  // slot is kept to the end, for body to read it again.
  auto each_tile = [&](bool warp_wide, bool hold, auto body) {
    if constexpr (kSplit) {
      body(own);
    } else {
      auto release = [&]() {
        if (warp_wide) __syncwarp();
        if (!warp_wide || lane == 0) mbar_arrive(&bars->work_empty[work_slot()]);
        ++taken;
      };
      for (;;) {
        bool ok = mbar_wait(&bars->work_full[work_slot()], work_phase(), ab, 0x3700u + work_slot());
        if (warp_wide) ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        const int4 w = bars->work[work_slot()];
        if (w.x < 0) break;
        if (!hold) release();
        if (!body(w)) break;
        asm volatile("" : "+r"(taken));  // (the slot's addresses are worked out again, not kept over the tile)
        if (hold) release();
      }
    }
  };

  if (kFuseDq && warp >= kDkvDrainWarp) {
    // ------------------------------------------------------------------ dQ drain (fused form)
    // Thread = q row of the pair's dQ tile (TMEM lane) x 64 head-dim columns, 32 at a time.
    setmaxnreg_dec<kFusedDrainRegs>();
    const int wq = warp & 3;
    const int half = (warp - kDkvDrainWarp) >> 2;
    // Columns 64 half .. + 63; with at most 64 of them in all, 32 half .. + 31.  (Where dq has 96 at most the last 32 hold zeros
    // and stay here.  Late scores are for more than 96, but asking for that at run time, with this test, keeps registers: causal 4 x 8192
    // 6941 us, 7004 with the other one, 7978 -> 8037 a whole pass with a constant.)
    const bool two = kLateS ? p.d_qk > 64 : p.dq_pairs > half;
    const int chunk = p.d_qk > 64 ? 2 * half : half;
    const uint32_t t_dq = tmem + ((uint32_t)(wq * 32) << 16) + kTile + chunk * 32;
    uint8_t* stage = ring + 3 * kTileBytes + (warp - kDkvDrainWarp) * kDqBlockBytes;
    const int n_q_tiles = p.q_len / kTile;
    bool ok = true;
    uint32_t n = 0;
    uint32_t v[32];
    // v -> the image: through the warp's own 4 KiB of shared memory, once what it held before has been read
    auto park = [&]() {
      if (lane == 0) bulk_wait_read();
      __syncwarp();
#pragma unroll
      for (int j = 0; j < 8; ++j)
        *reinterpret_cast<uint4*>(stage + j * 512 + lane * 16) = make_uint4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
    };
    auto send = [&](float* dst) {
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) bulk_reduce_add(dst, stage, kDqBlockBytes);
    };
    each_tile(true, false, [&](const int4& w) {
      const PartWalk<kSplit> walk = walk_of(w);
      const int4* entries = list_of(w);
      const uint32_t last = n + steps_of(w);
      for (int g = 0, o = walk.offset((int)rank); n < last && ok; ++g, o = offset_behind(o)) {
        // (w.y * group: batch * q heads + first q head of the group)
        float* head_base = p.dq_acc + ((int64_t)w.y * group + g) * n_q_tiles * (int64_t)kDqTileFloats +
                           (chunk * 4 + wq) * (kDqBlockBytes / 4);
        for (int e = walk.first(o); e < w.w && ok; e = walk.next(e), ++n) {
          float* dst = head_base + (int64_t)entries[e].x * kDqTileFloats;
          ok = mbar_wait(&bars->dq_full, n & 1u, ab, 0x3600u);
          ok = __all_sync(0xffffffffu, ok);
          if (!ok) break;
          tc_fence_after();
          tmem_ld32(t_dq, v);
          tmem_ld_wait();
          if (two) {
            park();
            tmem_ld32(t_dq + 32, v);
            if (kLateS) send(dst);
            tmem_ld_wait();
          }
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&bars->dq_free);
          if (two && !kLateS) send(dst);  // (dP^T waits for these columns more often: prefix 2 x 4096 618 -> 604 us)
          park();
          send(two ? dst + 4 * (kDqBlockBytes / 4) : dst);
        }
      }
      return ok;
    });
    if (lane == 0) bulk_wait_all();
  } else if (warp >= 16) {
   if constexpr (kFuseDq) setmaxnreg_dec<kFusedIssueRegs>();
   if (warp == kDkvTmaWarp) {
    if (elect_one()) {
      // tiles are two 64-column halves; with at most 64 real columns the second is never read
      const bool qk2 = p.d_qk > 64, v2 = p.d_v > 64;
      uint32_t n = 0;
      uint32_t stepped = 0;  // tiles with steps so far
      uint32_t asked = 0;
      bool ok = true;
      int4 w = own;
      while (ok) {
        if constexpr (!kSplit) {
          ok = mbar_wait(&bars->work_empty[work_slot()], work_phase() ^ 1u, ab, 0x3710u + work_slot());
          if (!ok) break;
          bars->work[work_slot()] = w;
          mbar_arrive(&bars->work_full[work_slot()]);
          ++taken;
          if (w.x < 0) break;
        }
        const PartWalk<kSplit> walk = walk_of(w);
        const int4* entries = list_of(w);
        const int kv_head = w.y % p.kv_heads, batch = w.y / p.kv_heads;
        const uint32_t first = n, last = n + steps_of(w);
        for (int g = 0, o = walk.offset((int)rank); n < last && ok; ++g, o = offset_behind(o)) {
          const int head = kv_head * group + g;
          const int64_t stat_base = ((int64_t)batch * p.q_heads + head) * p.q_len;
          for (int e = walk.first(o); e < w.w && ok; e = walk.next(e), ++n) {
            const int qt = entries[e].x;
            {
              const uint32_t s = 2u * (n & 1u);
              ok = mbar_wait(&bars->ring_empty[s], ((n >> 1) & 1u) ^ 1u, ab, 0x3100u + s);
              if (!ok) break;
              uint8_t* dst = ring + s * kTileBytes;
              if (kSplit) bars->step[s / 2] = entries[e];
              mbar_arrive_expect_tx(&bars->ring_full[s], (qk2 ? kTileBytes : kHalfBytes) + 2 * kTile * 4);
              tma_load_4d(dst, &tm_q, &bars->ring_full[s], 0, qt * kTile, head, batch);
              if (qk2) tma_load_4d(dst + kHalfBytes, &tm_q, &bars->ring_full[s], 64, qt * kTile, head, batch);
              // the step's statistics ride on the Q slot's barrier
              float* sdst = stats + (s / 2) * 2 * kTile;
              bulk_load(sdst, p.nlse2 + stat_base + (int64_t)qt * kTile, kTile * 4, &bars->ring_full[s]);
              bulk_load(sdst + kTile, p.delta + stat_base + (int64_t)qt * kTile, kTile * 4, &bars->ring_full[s]);
            }
            if (n == first) {  // K and V of the tile, once the MMAs of the last one have read theirs
              if (stepped > 0) ok = mbar_wait(&bars->acc_done, (stepped - 1) & 1u, ab, 0x3120u);
              if (!ok) break;
              mbar_arrive_expect_tx(&bars->stat_full[0], qk2 ? kTileBytes : kHalfBytes);
              tma_load_4d(k_smem, &tm_k, &bars->stat_full[0], 0, w.x * kTile, kv_head, batch);
              if (qk2) tma_load_4d(k_smem + kHalfBytes, &tm_k, &bars->stat_full[0], 64, w.x * kTile, kv_head, batch);
              mbar_arrive_expect_tx(&bars->stat_full[1], v2 ? kTileBytes : kHalfBytes);
              tma_load_4d(v_smem, &tm_v, &bars->stat_full[1], 0, w.x * kTile, kv_head, batch);
              if (v2) tma_load_4d(v_smem + kHalfBytes, &tm_v, &bars->stat_full[1], 64, w.x * kTile, kv_head, batch);
              ++stepped;
            }
            {
              const uint32_t s = do_bar(n);
              ok = mbar_wait(&bars->ring_empty[s], do_phase(n) ^ 1u, ab, 0x3100u + s);
              if (!ok) break;
              uint8_t* dst = ring + do_offset(n);
              mbar_arrive_expect_tx(&bars->ring_full[s], v2 ? kTileBytes : kHalfBytes);
              tma_load_4d(dst, &tm_do, &bars->ring_full[s], 0, qt * kTile, head, batch);
              if (v2) tma_load_4d(dst + kHalfBytes, &tm_do, &bars->ring_full[s], 64, qt * kTile, head, batch);
            }
          }
        }
        if (kSplit || !ok) break;
        // The next tile.  Asked for when all of this one is on its way, and no earlier: what a CTA has taken over, no other
        // can take that is done before it.
        mbar_arrive_expect_tx(&bars->answer_full, 16);
        clc_request(bars->answer, &bars->answer_full);
        ok = mbar_wait(&bars->answer_full, asked & 1u, ab, 0x3720u);
        ++asked;
        const int block = ok ? clc_block(bars->answer) : -1;
        fence_proxy_async_smem();  // read before the next answer overwrites it
        w = block >= 0 ? tile_of((unsigned)block) : make_int4(-1, 0, 0, 0);
      }
    }
  } else if (warp == kDkvMmaWarp) {
    if (elect_one()) {
      constexpr uint32_t idesc_s = make_idesc_bf16(kTile, kTile, false, false);
      // N of the accumulating MMAs = the gradient's columns: 128, or 64 when the tensor has at most 64
      const uint32_t idesc_dv = make_idesc_bf16(kTile, p.d_v <= 64 ? 64 : kHeadDim, false, true);
      const uint32_t idesc_dk = make_idesc_bf16(kTile, p.d_qk <= 64 ? 64 : kHeadDim, false, true);
      const uint32_t k_addr = smem_u32(k_smem), v_addr = smem_u32(v_smem), ds_addr = smem_u32(ds_smem);
      const uint32_t ring_addr = smem_u32(ring);
      const uint32_t t_st = tmem, t_dpt = tmem + kTile, t_dk = tmem + 2 * kTile, t_dv = tmem + 3 * kTile;
      auto q_addr = [&](uint32_t n) { return ring_addr + 2 * (n & 1u) * kTileBytes; };
      auto do_addr = [&](uint32_t n) { return ring_addr + do_offset(n); };
      auto q_wait = [&](uint32_t n, uint32_t tag) { return mbar_wait(&bars->ring_full[2 * (n & 1u)], (n >> 1) & 1u, ab, tag); };
      auto do_wait = [&](uint32_t n, uint32_t tag) { return mbar_wait(&bars->ring_full[do_bar(n)], do_phase(n), ab, tag); };
      // D = A B^T with both operands K-major (head_dim contiguous), K = head_dim
      auto issue_score = [&](uint32_t d, SmemDesc da, uint32_t b0, int nk) {
        const SmemDesc db = make_smem_desc_sw128(b0, 16, 1024);
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          if (nk != 8 && k >= nk) break;  // head dims below 128: the remaining slices multiply zeros
          const uint32_t off = (k >> 2) * kHalfBytes + (k & 3) * 32;
          umma_ss(d, desc_at(da, off), desc_at(db, off), idesc_s, k > 0 ? 1u : 0u);
        }
      };
      // descriptors of the stationary operands, built once
      const SmemDesc k_desc = make_smem_desc_sw128(k_addr, 16, 1024), v_desc = make_smem_desc_sw128(v_addr, 16, 1024);
      const SmemDesc ds_desc = make_smem_desc_sw128(ds_addr, 16, 1024);
      // fused form: the same two tiles seen MN-major (rows are the MMA's K dimension)
      const uint32_t idesc_dq = make_idesc_bf16(kTile, p.d_qk <= 64 ? 64 : kHeadDim, true, true);
      const SmemDesc ds_mn_desc = make_smem_desc_sw128(ds_addr, kHalfBytes, 1024);
      const SmemDesc k_mn_desc = make_smem_desc_sw128(k_addr, kHalfBytes, 1024);
      uint32_t n = 0;      // steps so far
      uint32_t tiles = 0;  // tiles with steps so far
      auto next_scores = [&]() {
        if (!q_wait(n + 1, 0x3240u)) return false;
        issue_score(t_st, k_desc, q_addr(n + 1), p.nk_qk);
        tc_commit(&bars->st_full);
        return true;
      };
      each_tile(false, false, [&](const int4& w) {
      const uint32_t first = n, last = n + steps_of(w);
      if (first == last) return true;
      bool ok = mbar_wait(&bars->stat_full[0], tiles & 1u, ab, 0x3200u) && q_wait(n, 0x3210u);
      if (ok) {
        mma_issue_fence();
        issue_score(t_st, k_desc, q_addr(n), p.nk_qk);
        tc_commit(&bars->st_full);
      }
      ok = ok && mbar_wait(&bars->stat_full[1], tiles & 1u, ab, 0x3201u) && do_wait(n, 0x3211u);
      if (kFuseDq && n > 0) ok = ok && mbar_wait(&bars->dq_free, (n - 1) & 1u, ab, 0x3251u);
      if (ok) {
        mma_issue_fence();
        issue_score(t_dpt, v_desc, do_addr(n), p.nk_v);
        tc_commit(&bars->dpt_full);
      }
      // the outputs of the tile before have been read
      if (tiles > 0) ok = ok && mbar_wait(&bars->out_free, (tiles - 1) & 1u, ab, 0x3260u);
      ++tiles;
      for (; n < last && ok; ++n) {
        const uint32_t ph = n & 1u;
        const uint32_t q_slot = q_addr(n), do_slot = do_addr(n);
        const bool more = n + 1 < last, begun = n > first;
        ok = mbar_wait(&bars->p_full, ph, ab, 0x3220u);
        if (!ok) break;
        mma_issue_fence();
        // dV += P^T dO: A = packed bf16 P^T in TMEM (16 packed columns at the start of every
        // 32-column quarter), B = the dO tile read MN-major, K = 128 query rows in eight slices
        const SmemDesc do_mn = make_smem_desc_sw128(do_slot, kHalfBytes, 1024);
#pragma unroll
        for (int k = 0; k < 8; ++k)
          umma_ts(t_dv, t_st + (k >> 1) * 32 + (k & 1) * 8, desc_at(do_mn, k * 2048), idesc_dv,
                  (begun || k > 0) ? 1u : 0u);
        tc_commit(&bars->ring_empty[do_bar(n)]);
        if (more && !kLateS) {
          ok = next_scores();
          if (!ok) break;
        }
        ok = mbar_wait(&bars->ds_full, ph, ab, 0x3230u);
        if (!ok) break;
        mma_issue_fence();
        if constexpr (kFuseDq) {
          // dQ_partial = dS K over the dP^T columns (every compute warp has read dP^T(n) before it
          // arrived on ds_full): A = the dS^T tile read MN-major (M = q), B = the K tile read
          // MN-major (N = head dim), K = 128 kv rows in eight slices.  Issued ahead of dK so the
          // drain warps read it out while dK runs.
#pragma unroll
          for (int k = 0; k < 8; ++k)
            umma_ss(t_dpt, desc_at(ds_mn_desc, k * 2048), desc_at(k_mn_desc, k * 2048), idesc_dq, k > 0 ? 1u : 0u);
          tc_commit(&bars->dq_full);
          if (more && kLateS) {
            ok = next_scores();
            if (!ok) break;
          }
        }
        // dK += dS^T Q: A = dS^T from shared memory (K-major, two 64-column halves), B = the Q
        // tile read MN-major
        const SmemDesc q_mn = make_smem_desc_sw128(q_slot, kHalfBytes, 1024);
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const uint32_t off = (k >> 2) * kHalfBytes + (k & 3) * 32;
          umma_ss(t_dk, desc_at(ds_desc, off), desc_at(q_mn, k * 2048), idesc_dk, (begun || k > 0) ? 1u : 0u);
        }
        tc_commit(&bars->ds_free);
        tc_commit(&bars->ring_empty[2 * (n & 1)]);
        if (more) {
          ok = do_wait(n + 1, 0x3241u);
          if (!ok) break;
          if constexpr (kFuseDq) {  // the dP^T columns still hold dQ_partial(n) until it is drained
            ok = mbar_wait(&bars->dq_free, ph, ab, 0x3250u);
            if (!ok) break;
            mma_issue_fence();
          }
          issue_score(t_dpt, v_desc, do_addr(n + 1), p.nk_v);
          tc_commit(&bars->dpt_full);
        }
      }
      tc_commit(&bars->acc_done);
      return ok;
      });
    }
   }
  } else {
    // 16 warps on one 128 x 128 tile: a warp has 32 kv rows (TMEM lanes) x one 32-column quarter, which its threads hold as
    // matrix fragments (tmem_ld_frag): four rows x eight columns each.  The statistics belong to columns.  With a row
    // and 32 columns a thread, every warp read 32 columns' pairs in 16 LDS.128, all lanes the same address: 837 of some
    // 4600 cycles a step of the shared-memory data pipe, which the kernel kept 99 % busy (MMAs 51 %, loads and stores 48 %).
    // In fragments they are eight LDS.64, and dS^T goes out by stmatrix without bank conflicts.  A row a thread -> this,
    // us a pass: 4 x 8192, 32 / 8 6977 -> 6860, 8 x 16384, 16 heads, window 4096 6315 -> 6118, 4 x 2048, 16 / 16 330 -> 313,
    // 2 x 8192, 16 / 4, d 64 1209 -> 1185, repeatable 2 x 4096, 16 / 1 496 -> 480, soft cap 4 x 4096, 16 / 8, window 768
    // 641 -> 589.
    if constexpr (kFuseDq) setmaxnreg_inc<kFusedComputeRegs>();
    const int cq = warp >> 2;      // column quarter 0..3
    const int wq = warp & 3;       // TMEM lane quarter
    const int r = wq * 32 + lane;  // kv row within the tile
    const bool has_seg = p.q_seg != nullptr;
    const uint32_t lane_addr = (uint32_t)(wq * 32) << 16;
    const uint32_t t_st = tmem + lane_addr + cq * 32;
    const uint32_t t_dpt = tmem + lane_addr + kTile + cq * 32;
    // Element at(k, hq) + u: kv row row0 + 8 hq, q column col0 + 8 k + u of the quarter.
    auto at = [](int k, int hq) { return 16 * (hq >> 1) + 4 * k + 2 * (hq & 1); };
    const int row0 = wq * 32 + (lane >> 2);
    const int col0 = 2 * (lane & 3);
    // dS^T rows row.., columns cq*32 .. +31: 64 bytes = four 16-byte chunks of the row's 128-byte
    // segment in swizzle half cq / 2; chunk c sits at position c ^ (row mod 8).  Lane: row lane % 8, chunk lane / 8.
    const uint32_t ds_addr = smem_u32(ds_smem) + (cq >> 1) * kHalfBytes + (wq * 32 + (lane & 7)) * 128 +
                             ((((cq & 1) * 4 + (lane >> 3)) ^ (lane & 7)) << 4);
    const float c = kSoftCap ? p.soft_cap * kLog2e : p.scale_log2;
    uint32_t n = 0;      // steps so far
    uint32_t tiles = 0;  // tiles with steps so far
    each_tile(true, true, [&](const int4& w) {
    const int kv_row = w.x * kTile + row0;
    const int32_t* kv_seg_row = has_seg ? p.kv_seg + (int64_t)(w.y / p.kv_heads) * p.kv_len + kv_row : nullptr;
    const int32_t* q_seg_row = has_seg ? p.q_seg + (int64_t)(w.y / p.kv_heads) * p.q_len : nullptr;
    const int4* entries = list_of(w);
    const int ebeg = w.z, eend = w.w;
    const uint32_t first = n, last = n + steps_of(w);
    bool ok = true;

    // (kSplit: one run through this CTA's steps, whose entries the TMA warp leaves in shared memory)
    while (n < last && ok) {
      int4 ent_next = make_int4(0, 0, 0, 0);
      if constexpr (!kSplit) ent_next = entries[ebeg];
      for (int e = ebeg; (kSplit ? n < last : e < eend) && ok; ++e, ++n) {
        int4 ent = ent_next;
        if (!kSplit && e + 1 < eend) ent_next = entries[e + 1];
        const uint32_t ph = n & 1u;
        const uint32_t itq = 2u * n;
        ok = mbar_wait(&bars->ring_full[itq % kBwdStages], (itq / kBwdStages) & 1u, ab, 0x3420u);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        if constexpr (kSplit) ent = bars->step[(itq % kBwdStages) / 2];
        const int st = ent.y & 3;
        const int q0 = ent.x * kTile + cq * 32 + col0;  // first q column of this thread
        // columns 8 k + 0, 1: word 4 k
        const float2* nl2 = reinterpret_cast<const float2*>(stats + ((itq % kBwdStages) / 2) * 2 * kTile + cq * 32 + col0);
        const float2* dl2 = nl2 + kTile / 2;
        // table: a lane reads eight columns of its four rows and keeps a bit for each of them, row by row (two columns at a
        // time, as they are used, took 16 loads: prefix 2 x 4096, 16 / 4 631 us a pass instead of 577)
        uint32_t mask_bits = 0;
        if (st == 1 && p.fn.kind == SPLASH_MASK_TABLE) {
          const int8_t* mrow = p.pmb + ((int64_t)ent.z * p.pm_bkv + (kv_row % p.pm_bkv)) * p.pm_bq +
                               ((ent.x * kTile + cq * 32) % p.pm_bq) + 8 * (lane & 3);
#pragma unroll
          for (int hq = 0; hq < 4; ++hq) {
            const int2 m = __ldg(reinterpret_cast<const int2*>(mrow + (int64_t)(8 * hq) * p.pm_bq));
            mask_bits |= (nonzero_bytes((uint32_t)m.x) | nonzero_bytes((uint32_t)m.y) << 4) << (8 * hq);
          }
        }

        ok = mbar_wait(&bars->st_full, ph, ab, 0x3400u);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        tc_fence_after();
        float pr[32];
        {
          uint32_t v[32];
          tmem_ld_frag(t_st, v);
          tmem_ld_frag(t_st + kLanes16, v + 16);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 32; ++j) pr[j] = __uint_as_float(v[j]);
        }
        // Soft cap: tiles without a mask take tanh beside the exponentials (one pass behind the other keeps the FMA units waiting
        // for the special-function ones and these for them)
        bool beside = false;
        if constexpr (kSoftCap) {
          const bool small = tanh_is_small(pr, p.softcap_a);
          beside = small && st != 1 && !(has_seg && !((ent.y >> 4) & 1));
          if (!beside) tanh_all(pr, p.softcap_a, small);
        }
        if (st == 1) {
          if (p.fn.kind != SPLASH_MASK_TABLE) {
#pragma unroll
            for (int k = 0; k < 4; ++k)
#pragma unroll
              for (int u = 0; u < 2; ++u) {
                const int q = q0 + 8 * k + u;
                const RowInterval iv = mask_fn_interval(p.fn, p.q_sequence == nullptr ? q : __ldg(p.q_sequence + q));
#pragma unroll
                for (int hq = 0; hq < 4; ++hq)
                  if (kv_row + 8 * hq < iv.lo || kv_row + 8 * hq > iv.hi) pr[at(k, hq) + u] = kMaskedLogit;
              }
          } else {
#pragma unroll
            for (int k = 0; k < 4; ++k) {  // lane 4 i + k of the four that share the rows holds columns 8 k .. + 7
              const uint32_t mine = __shfl_sync(0xffffffffu, mask_bits, k, 4) >> col0;
#pragma unroll
              for (int hq = 0; hq < 4; ++hq)
#pragma unroll
                for (int u = 0; u < 2; ++u)
                  if (((mine >> (8 * hq + u)) & 1u) == 0u) pr[at(k, hq) + u] = kMaskedLogit;
            }
          }
        }
        if (has_seg && !((ent.y >> 4) & 1)) {  // (bit set: the whole tile lies inside one segment)
          int kv_seg[4];
#pragma unroll
          for (int hq = 0; hq < 4; ++hq) kv_seg[hq] = __ldg(kv_seg_row + 8 * hq);
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const int2 sv = __ldg(reinterpret_cast<const int2*>(q_seg_row + q0) + 4 * k);
#pragma unroll
            for (int hq = 0; hq < 4; ++hq) {
              if (sv.x != kv_seg[hq]) pr[at(k, hq)] = kMaskedLogit;
              if (sv.y != kv_seg[hq]) pr[at(k, hq) + 1] = kMaskedLogit;
            }
          }
        }
        auto send_p = [&](const uint32_t (&pk)[16]) {
          tmem_st_frag(t_st, pk);
          tmem_st_frag(t_st + kLanes16, pk + 8);
          tmem_st_wait();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&bars->p_full);
        };
        if (kSoftCap && beside) {
          uint32_t pk[16];
          const float2 a2 = make_float2(p.softcap_a, p.softcap_a), c2 = make_float2(c, c);
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const float2 nl = nl2[4 * k];
#pragma unroll
            for (int hq = 0; hq < 4; ++hq) {
              const int j = at(k, hq);
              const float2 th = tanh_small(__fmul2_rn(make_float2(pr[j], pr[j + 1]), a2));
              const float2 x = __ffma2_rn(th, c2, nl);
              const float p0 = ex2(x.x), p1 = ex2(x.y);
              pk[j / 2] = pack_bf16(p0, p1);
              pr[j] = p0 * fmaf(-th.x, th.x, 1.0f);
              pr[j + 1] = p1 * fmaf(-th.y, th.y, 1.0f);
            }
          }
          send_p(pk);
        } else {
          uint32_t pk[16];
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const float2 nl = nl2[4 * k];
#pragma unroll
            for (int hq = 0; hq < 4; ++hq) {
              const int j = at(k, hq);
              const float2 th = make_float2(fmaxf(pr[j], -1.0f), fmaxf(pr[j + 1], -1.0f));
              const float2 x = __ffma2_rn(make_float2(pr[j], pr[j + 1]), make_float2(c, c), nl);
              pr[j] = ex2(x.x);
              pr[j + 1] = ex2(x.y);
              pk[j / 2] = pack_bf16(pr[j], pr[j + 1]);
              if constexpr (kSoftCap) {
                pr[j] *= fmaf(-th.x, th.x, 1.0f);
                pr[j + 1] *= fmaf(-th.y, th.y, 1.0f);
              }
            }
          }
          send_p(pk);
        }
        ok = mbar_wait(&bars->dpt_full, ph, ab, 0x3410u);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        tc_fence_after();
        uint32_t pk[16];
        {
          uint32_t v[32];
          tmem_ld_frag(t_dpt, v);
          tmem_ld_frag(t_dpt + kLanes16, v + 16);
          tmem_ld_wait();
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const float2 nd = dl2[4 * k];  // -di of the two query columns
#pragma unroll
            for (int hq = 0; hq < 4; ++hq) {
              const int j = at(k, hq);
              const float2 a = __fmul2_rn(make_float2(pr[j], pr[j + 1]),
                                          __fadd2_rn(make_float2(__uint_as_float(v[j]), __uint_as_float(v[j + 1])), nd));
              pk[j / 2] = pack_bf16(a.x, a.y);
            }
          }
        }
        if (n > 0) {  // the previous step's dK must have finished reading the tile
          ok = mbar_wait(&bars->ds_free, (n - 1) & 1u, ab, 0x3430u);
          ok = __all_sync(0xffffffffu, ok);
          if (!ok) break;
        }
#pragma unroll
        for (int hq = 0; hq < 4; ++hq) {
          const int j = 8 * (hq >> 1) + (hq & 1);
          stmatrix_x4(ds_addr + hq * 1024, pk[j], pk[j + 2], pk[j + 4], pk[j + 6]);
        }
        fence_proxy_async_smem();  // generic-proxy stores -> visible to the MMA's async-proxy reads
        __syncwarp();
        if (lane == 0) mbar_arrive(&bars->ds_full);
      }
    }

    // epilogue: dK (scaled) and dV, 32 columns per thread
    {  // (the tile's place is read again: the loop over the steps needs the registers)
    const int4 again = kSplit ? own : ld_again(&bars->work[work_slot()]);
    const int batch = again.y / p.kv_heads, kv_head = again.y % p.kv_heads, kv_row = again.x * kTile + r;
    const uint32_t n_steps = last - first;
    __nv_bfloat16* dk = p.out0 + (int64_t)batch * p.out0_sb + (int64_t)kv_head * p.out0_sh +
                        (int64_t)kv_row * p.out0_ss + cq * 32;
    __nv_bfloat16* dv = p.out1 + (int64_t)batch * p.out1_sb + (int64_t)kv_head * p.out1_sh +
                        (int64_t)kv_row * p.out1_ss + cq * 32;
    if constexpr (kSplit) {
      if (n_steps > 0 && ok) {
        ok = mbar_wait(&bars->acc_done, 0, ab, 0x3500u);
        ok = __all_sync(0xffffffffu, ok);
      }
      float4* part = reinterpret_cast<float4*>(smem) + r;
      if (ok) {
        tc_fence_after();
#pragma unroll
        for (int which = 0; which < 2; ++which) {  // dk, dv: columns cq * 32 .. + 31
          uint32_t v[32];
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] = 0u;
          if (n_steps > 0) {
            tmem_ld32(tmem + lane_addr + (2 + which) * kTile + cq * 32, v);
            tmem_ld_wait();
          }
#pragma unroll
          for (int j = 0; j < 8; ++j)
            part[(which * (kHeadDim / 4) + cq * 8 + j) * kTile] =
                make_float4(__uint_as_float(v[4 * j]), __uint_as_float(v[4 * j + 1]), __uint_as_float(v[4 * j + 2]),
                            __uint_as_float(v[4 * j + 3]));
        }
      }
      tc_fence_before();
      cluster_sync();  // (with the same call of the other warps below)
      bool good = true;
      for (int s = 0; s < p.n_split; ++s) good = good && cluster_ld_u32(cluster_addr(&bars->abort_flag, s)) == 0u;
      if (good) {
        // groups of eight columns (16 of dk, 16 of dv) shared out over the cluster's warps; lane = row
        for (int c = (int)rank * 4 + cq; c < 2 * kHeadDim / 8; c += 4 * p.n_split) {
          const int which = c / (kHeadDim / 8), col = (c % (kHeadDim / 8)) * 8;
          if (col >= (which ? p.d_v : p.d_qk)) continue;
          float4 x = make_float4(0.f, 0.f, 0.f, 0.f), y = x;
          for (int s = 0; s < p.n_split; ++s) {
            const float4 u = cluster_ld_v4(cluster_addr(part + (2 * c) * kTile, s));
            const float4 w = cluster_ld_v4(cluster_addr(part + (2 * c + 1) * kTile, s));
            x.x += u.x, x.y += u.y, x.z += u.z, x.w += u.w;
            y.x += w.x, y.y += w.y, y.z += w.z, y.w += w.w;
          }
          const float mul = which ? 1.0f : p.scale;
          const uint4 w = make_uint4(pack_bf16(x.x * mul, x.y * mul), pack_bf16(x.z * mul, x.w * mul),
                                     pack_bf16(y.x * mul, y.y * mul), pack_bf16(y.z * mul, y.w * mul));
          const SplashPeerOutput& peer = which ? p.out1_peer : p.out0_peer;
          *reinterpret_cast<uint4*>((which ? dv : dk) - cq * 32 + col) = w;
          if (peer.ptrs) *reinterpret_cast<uint4*>(peer_row(peer, batch, kv_head, kv_row) + col) = w;
        }
      }
    } else {
      if (n_steps > 0 && ok) {
        ok = mbar_wait(&bars->acc_done, tiles++ & 1u, ab, 0x3500u);
        ok = __all_sync(0xffffffffu, ok);
      }
      if (ok) {
        tc_fence_after();
        // (context parallelism: the rows also go to the ranks that own them in the sequence-sharded layout)
#pragma unroll
        for (int which = 0; which < 2; ++which) {
          uint32_t v[32];
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] = 0u;  // (a kv tile that no step touches gets zeros)
          if (n_steps > 0) {
            tmem_ld32(tmem + lane_addr + (2 + which) * kTile + cq * 32, v);
            tmem_ld_wait();
          }
          if (which == 1 && n_steps > 0) {
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&bars->out_free);
          }
          const int64_t ss = which ? p.out1_ss : p.out0_ss;
          store_rows32_peer((which ? dv : dk) - cq * 32 - (int64_t)lane * ss, ss, which ? p.out1_peer : p.out0_peer, batch, kv_head,
                            kv_row - lane, v, which ? 1.0f : p.scale, cq * 32, which ? p.d_v : p.d_qk);
        }
      }
    }
    }
    return ok;
    });
  }

  if constexpr (kSplit) {
    if (warp >= 16) cluster_sync();  // the parts are in place
    cluster_sync();                  // they have been read
  }
  tc_fence_before();
  __syncthreads();
  if (warp == kDkvMmaWarp) {
    __syncwarp();
    drain_after_give_up(&bars->abort_flag);
    tmem_dealloc(tmem, 512);
  }
}

// ------------------------------------------------------------------------------------------
// fused form: fp32 dQ image -> bf16 dQ
// ------------------------------------------------------------------------------------------
// One CTA per 128 x 128 tile, a warp for 32 rows x 64 columns: a warp instruction reads 512 bytes of the image in one
// piece (lane = row, as the rows came from TMEM) and writes 64-byte runs of eight bf16 rows; HBM-bound: 16 + 8 bytes for
// four columns of a row.  32768 rows x 32 117 us = 6.9 TB/s, 1.05 of the measured copy rate (139 with 64-byte reads);
// 32768 x 128 at a window: 314 -> 233.  Chunks beyond dq's columns are neither cleared nor read: 2 x 8192, 16 heads, d 64
// 1243 -> 1216 us a pass.
struct DqConvertParams {
  const float* acc;
  __nv_bfloat16* dq;
  int64_t dq_sb, dq_sh, dq_ss;
  int q_heads, n_q_tiles;
  int d_qk;  // columns of dq
  float scale;
  SplashPeerOutput dq_peer;  // second destination in other ranks' memory (ptrs == nullptr: none)
};

__global__ void __launch_bounds__(256) splash_dq_convert_kernel(const DqConvertParams p) {
  const int64_t tile = blockIdx.x;
  const int qt = (int)(tile % p.n_q_tiles);
  const int64_t bh = tile / p.n_q_tiles;
  const int h = (int)(bh % p.q_heads);
  const int64_t b = bh / p.q_heads;
  const int wq = (threadIdx.x >> 5) & 3, half = threadIdx.x >> 7, lane = threadIdx.x & 31;
  const int row = qt * kTile + wq * 32;
  const uint4* src = reinterpret_cast<const uint4*>(p.acc + tile * kDqTileFloats) + lane;
  uint4 x[2][8];
#pragma unroll
  for (int c = 0; c < 2; ++c)
    if ((half * 2 + c) * 32 < p.d_qk)
#pragma unroll
      for (int j = 0; j < 8; ++j) x[c][j] = __ldcs(src + (((half * 2 + c) * 4 + wq) * 8 + j) * 32);
  __nv_bfloat16* row0 = p.dq + b * p.dq_sb + h * p.dq_sh + (int64_t)row * p.dq_ss;
#pragma unroll
  for (int c = 0; c < 2; ++c) {
    const int col0 = (half * 2 + c) * 32;
    if (col0 >= p.d_qk) break;
    uint32_t v[32];
#pragma unroll
    for (int j = 0; j < 8; ++j) v[4 * j] = x[c][j].x, v[4 * j + 1] = x[c][j].y, v[4 * j + 2] = x[c][j].z, v[4 * j + 3] = x[c][j].w;
    store_rows32_peer(row0, p.dq_ss, p.dq_peer, (int)b, h, row, v, p.scale, col0, p.d_qk);
  }
}

// ------------------------------------------------------------------------------------------
// host launcher
// ------------------------------------------------------------------------------------------
size_t bwd_workspace_bytes(int64_t batch, int64_t q_heads, int64_t q_len) {
  if (batch <= 0 || q_heads <= 0 || q_len <= 0) return 0;
  const size_t n = (size_t)batch * (size_t)q_heads * (size_t)q_len * sizeof(float);
  return 2 * ((n + 255) & ~(size_t)255);  // di, then -logsumexp * log2(e)
}
// Fused form: the same two per-row arrays, then the fp32 dQ image.
size_t bwd_fused_workspace_bytes(int64_t batch, int64_t q_heads, int64_t q_len) {
  const size_t base = bwd_workspace_bytes(batch, q_heads, q_len);
  if (base == 0) return 0;
  return base + (size_t)batch * (size_t)q_heads * (size_t)q_len * kHeadDim * sizeof(float);
}

using DkvKernel = void (*)(CUtensorMap, CUtensorMap, CUtensorMap, CUtensorMap, BwdParams);
static DkvKernel dkv_kernel_for(bool split, bool fused, bool soft_cap, bool late) {
  static const DkvKernel kernels[2][2][2] = {
      {{splash_dkv_kernel<false, false, false, false>, splash_dkv_kernel<true, false, false, false>},
       {splash_dkv_kernel<false, true, false, false>, splash_dkv_kernel<true, true, false, false>}},
      {{splash_dkv_kernel<false, false, true, false>, splash_dkv_kernel<true, false, true, false>},
       {splash_dkv_kernel<false, true, true, false>, splash_dkv_kernel<true, true, true, false>}}};
  if (late) return split ? splash_dkv_kernel<false, true, true, true> : splash_dkv_kernel<false, true, false, true>;
  return kernels[split][fused][soft_cap];
}
// Whether S^T of the next step is issued behind dQ of this one instead of behind dV.  Whole backward, d 128: causal 4 x 8192,
// 32 / 8 heads 5580 -> 5465 us, 2 x 4096 787 -> 759, 4 x 2048, 16 / 16 265 -> 257; full 1 x 4096, 32 / 8 710 -> 691; window 4096,
// 8 x 16384, 16 / 16 10717 -> 10482.  d 104 .. 120 take the same time either way (causal 2 x 8192, 16 / 4 1354 1360, 1338 1344, 1387 1392).
// Up to 96 the drain sends three quarters or half of dQ, and there is less to run the scores under: d 96 1164 -> 1265, d 80
// 1097 -> 1192, d 72 1131 -> 1245, d 64 802 -> 984.  A soft cap, whose P^T takes longer to form, wants its scores early
// (3 x 1664, 12 / 4, d 80, window 768 89 -> 95, causal 4 x 4096, 16 / 8 738 -> 781); partial blocks read from a table did, but no
// longer do (prefix 2 x 4096, 16 / 4 394 -> 380, 4 x 1024, 32 / 8 163 -> 159, 8192, 16 / 16, d 96 707 -> 694) and are left as they are.
// Without dQ there is nothing to put them behind (4 x 4096, 16 / 8: behind dS^T's arrival 1097 -> 1158).
static bool late_scores(const SplashBwdArgs& a, bool fused) {
  const bool table = a.mask_fn.kind == SPLASH_MASK_TABLE && a.sched_dkv.partial_mask_blocks != nullptr;
  return fused && a.soft_cap == 0.f && a.q.size[3] > 96 && !table;
}

// The groups of a dkv launch that come chunk by chunk; the others are its last chunk.  A chunk's rows fill the SMs only
// while the next chunk follows; behind the last one they wait for its longest row, which in a triangle of rows takes as
// long as several chunks of one group together.  So the last chunk has groups enough for a row an SM, longest first over
// all of them (prefix mask 2 x 4096, 16 / 4 heads, 8 groups of 32 rows: 682 -> 617 us a pass; causal 4 x 8192, 32 / 8:
// 7302 -> 7243; two or four rows an SM: 617 and 7284 .. 7527, the dQ images of those groups no longer stay in L2).
static int last_chunk(int64_t n_groups, int64_t chunk_groups, int64_t n_rows) {
  const int64_t last = (kSms + n_rows - 1) / n_rows;
  return n_groups > last ? (int)((n_groups - last) / chunk_groups * chunk_groups) : 0;
}

// CTAs that share a kv tile of this call's dkv kernel (head dims up to 128)
static int dkv_split(const SplashBwdArgs& a, const SplashShards& shards, bool fused, const int32_t* clusters) {
  if (a.q_segment_ids != nullptr || a.q_sequence != nullptr) return 1;
  // a shard of the query rows: its dk / dv are one summand of the call's, there are no bits to keep; where the
  // mask is a function, the first shard (whose rows need no q_sequence) leaves its kv tiles whole as the others do
  if (shards.q_shards > 1 && a.mask_fn.kind != SPLASH_MASK_TABLE) return 1;
  const int64_t n_rows = a.k.size[2] / kTile;
  RowWork rw = estimate_row_work(a.mask_fn, (int)n_rows, kTile, (int)(a.q.size[2] / kTile),
                                 n_rows * a.k.size[0] * a.k.size[1] * (shards.head_shards > 1 ? shards.head_shards : 1), true);
  rw.scale((int)(a.q.size[1] / a.k.size[1]));  // a kv tile walks every q head of its group
  const bool soft_cap = a.soft_cap != 0.f, late = late_scores(a, fused);
  return row_parts(rw, clusters, [&] {
    return cluster_capacity((const void*)dkv_kernel_for(true, fused, soft_cap, late),
                            4 + (soft_cap ? 1 : 0) + (fused ? 2 : 0) + (late ? 4 : 0),
                            fused ? kFusedThreads : kDkvThreads, kDkvSmemBytes);
  });
}

int bwd_row_parts(const SplashBwdArgs& a, const SplashShards& shards, const int32_t* clusters) {
  for (int i = 0; i < 4; ++i)
    if (a.q.size[i] <= 0 || a.k.size[i] <= 0 || a.v.size[i] <= 0) return SPLASH_ERR_INVALID_ARGUMENT;
  if (a.q.size[2] % kTile != 0 || a.k.size[2] % kTile != 0) return SPLASH_ERR_INVALID_ARGUMENT;
  if (a.mask_fn.kind == SPLASH_MASK_CHUNKED && a.mask_fn.chunk <= 0) return SPLASH_ERR_INVALID_ARGUMENT;
  if (a.q.size[3] > kHeadDim || a.v.size[3] > kHeadDim) return 1;
  return dkv_split(a, shards, (a.flags & SPLASH_BWD_FUSED_DQ) != 0, clusters);
}

int launch_bwd(const SplashBwdArgs& a, const SplashShards& shards, cudaStream_t stream) {
  int st;
  const SplashTensor* ts[8] = {&a.q, &a.k, &a.v, &a.o, &a.d_o, &a.dq, &a.dk, &a.dv};
  for (int i = 0; i < 8; ++i)
    if ((st = check_bf16_tensor(*ts[i]))) return st;
  const int64_t B = a.q.size[0], Hq = a.q.size[1], Sq = a.q.size[2], D = a.q.size[3];
  const int64_t Hkv = a.k.size[1], Skv = a.k.size[2];
  // head dims below 128 are read in place (zero-extended by the TMA boxes), see splash_fwd
  const int64_t Dv = a.v.size[3];
  // head dims above 128 (up to 256): passes of their own, splash_bwd_wide_sm100.cu
  if (D > 2 * kHeadDim || Dv > 2 * kHeadDim) return SPLASH_ERR_UNSUPPORTED;
  const bool wide = D > kHeadDim || Dv > kHeadDim;
  if (D % 8 != 0 || Dv % 8 != 0) return SPLASH_ERR_INVALID_ARGUMENT;
  auto same3 = [](const SplashTensor& x, const SplashTensor& y) {
    return x.size[0] == y.size[0] && x.size[1] == y.size[1] && x.size[2] == y.size[2];
  };
  if (!same3(a.q, a.o) || !same3(a.q, a.d_o) || !same3(a.q, a.dq) || !same3(a.k, a.v) || !same3(a.k, a.dk) ||
      !same3(a.k, a.dv) || a.k.size[0] != B || a.k.size[3] != D || a.dq.size[3] != D || a.dk.size[3] != D ||
      a.o.size[3] != Dv || a.d_o.size[3] != Dv || a.dv.size[3] != Dv)
    return SPLASH_ERR_INVALID_ARGUMENT;
  if (Hkv <= 0 || Hq % Hkv != 0) return SPLASH_ERR_INVALID_ARGUMENT;
  if (Sq % kTile != 0 || Skv % kTile != 0) return SPLASH_ERR_INVALID_ARGUMENT;
  if ((a.q_segment_ids == nullptr) != (a.kv_segment_ids == nullptr))
    return SPLASH_ERR_INVALID_ARGUMENT;
  if (a.logsumexp == nullptr || a.error_record == nullptr || a.workspace == nullptr)
    return SPLASH_ERR_INVALID_ARGUMENT;
  const bool fused = (a.flags & SPLASH_BWD_FUSED_DQ) != 0 && !wide;  // the wide passes are separate by construction
  if ((st = check_peer_output(a.dq_peer, Sq, D)) || (st = check_peer_output(a.dk_peer, Skv, D)) ||
      (st = check_peer_output(a.dv_peer, Skv, Dv)))
    return st;
  if ((a.dq_peer.ptrs || a.dk_peer.ptrs || a.dv_peer.ptrs) && !fused) return SPLASH_ERR_UNSUPPORTED;
  if (a.workspace_bytes < (fused ? bwd_fused_workspace_bytes(B, Hq, Sq) : bwd_workspace_bytes(B, Hq, Sq)))
    return SPLASH_ERR_INVALID_ARGUMENT;
  if ((reinterpret_cast<uintptr_t>(a.workspace) & 255u) != 0) return SPLASH_ERR_INVALID_ARGUMENT;
  if (a.sched_dkv.row_ptr == nullptr || a.sched_dkv.entries == nullptr || a.sched_dkv.n_rows != Skv / kTile)
    return SPLASH_ERR_INVALID_ARGUMENT;
  if (!fused && (a.sched_dq.row_ptr == nullptr || a.sched_dq.entries == nullptr || a.sched_dq.n_rows != Sq / kTile))
    return SPLASH_ERR_INVALID_ARGUMENT;  // the fused form walks the dkv schedule only
  if (a.mask_fn.kind == SPLASH_MASK_CHUNKED && a.mask_fn.chunk <= 0)
    return SPLASH_ERR_INVALID_ARGUMENT;
  if (Hq > 65535 || B > 65535 || Sq / kTile > 65535 || Skv / kTile > 65535) return SPLASH_ERR_TOO_LARGE;
  if (!(a.scale > 0.f) || !(a.scale < 1.0e30f)) return SPLASH_ERR_INVALID_ARGUMENT;

  CUtensorMap tm_q, tm_do, tm_k, tm_v;
  const int box_rows = wide ? kSub : kTile;
  if ((st = make_tile_tensor_map(&tm_q, a.q, box_rows)) || (st = make_tile_tensor_map(&tm_do, a.d_o, box_rows)) ||
      (st = make_tile_tensor_map(&tm_k, a.k, box_rows)) || (st = make_tile_tensor_map(&tm_v, a.v, box_rows)))
    return st;

  const uint32_t mask = a.launch_mask == 0 ? 7u : a.launch_mask;
  float* delta = static_cast<float*>(a.workspace);
  float* nlse2 = reinterpret_cast<float*>(static_cast<uint8_t*>(a.workspace) + bwd_workspace_bytes(B, Hq, Sq) / 2);
  float* dq_acc = reinterpret_cast<float*>(static_cast<uint8_t*>(a.workspace) + bwd_workspace_bytes(B, Hq, Sq));
  // (fused form: the image the reductions add into starts at zero; the di pass clears it while it streams)
  if (mask & 1u) {
    DeltaParams dp;
    dp.o = static_cast<const __nv_bfloat16*>(a.o.data);
    dp.d_o = static_cast<const __nv_bfloat16*>(a.d_o.data);
    dp.o_sb = a.o.stride[0];
    dp.o_sh = a.o.stride[1];
    dp.o_ss = a.o.stride[2];
    dp.do_sb = a.d_o.stride[0];
    dp.do_sh = a.d_o.stride[1];
    dp.do_ss = a.d_o.stride[2];
    dp.delta = delta;
    dp.lse = a.logsumexp;
    dp.nlse2 = nlse2;
    dp.q_heads = (int)Hq;
    dp.q_len = (int)Sq;
    dp.d_v = (int)Dv;
    dp.dq_image = fused ? dq_acc : nullptr;
    dp.dq_chunks = (int)((D + 31) / 32);
    const unsigned blocks = (unsigned)(B * Hq * Sq / kDeltaRowsPerBlock);
    splash_delta_kernel<<<blocks, 256, 0, stream>>>(dp);
    if (cudaGetLastError() != cudaSuccess) return SPLASH_ERR_CUDA;
  }

  const bool soft_cap = a.soft_cap != 0.f;
  if (soft_cap && !(a.soft_cap > 0.f)) return SPLASH_ERR_INVALID_ARGUMENT;
  auto* dq_kernel = soft_cap ? splash_dq_kernel<true> : splash_dq_kernel<false>;
  const bool late = late_scores(a, fused);
  DkvKernel dkv_kernel = dkv_kernel_for(false, fused, soft_cap, late);
  const int dkv_smem = kDkvSmemBytes;
  // function attributes are per device: remember which devices have been set up
  {
    static std::mutex attr_mu;
    static bool attr_done[64][8] = {};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return SPLASH_ERR_CUDA;
    std::lock_guard<std::mutex> lock(attr_mu);
    bool& done = attr_done[dev][(soft_cap ? 1 : 0) + (fused ? 2 : 0) + (late ? 4 : 0)];
    if (!done) {
      if (cudaFuncSetAttribute(dq_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kDqSmemBytes) !=
              cudaSuccess ||
          cudaFuncSetAttribute(dkv_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, dkv_smem) != cudaSuccess)
        return SPLASH_ERR_CUDA;
      done = true;
    }
  }

  BwdParams p;
  p.out0_peer = SplashPeerOutput{};
  p.out1_peer = SplashPeerOutput{};
  p.nlse2 = nlse2;
  p.delta = delta;
  p.q_seg = a.q_segment_ids;
  p.kv_seg = a.kv_segment_ids;
  p.q_sequence = a.q_sequence;
  p.fn = a.mask_fn;
  p.q_len = (int)Sq;
  p.kv_len = (int)Skv;
  p.q_heads = (int)Hq;
  p.kv_heads = (int)Hkv;
  p.d_qk = (int)D;
  p.d_v = (int)Dv;
  p.nk_qk = (int)((D + 15) / 16);
  p.nk_v = (int)((Dv + 15) / 16);
  p.scale = a.scale;
  p.scale_log2 = a.scale * kLog2e;
  p.err = a.error_record;
  p.soft_cap = a.soft_cap;
  p.softcap_a = soft_cap ? a.scale / a.soft_cap : 0.f;
  p.dq_acc = fused ? dq_acc : nullptr;
  p.dq_pairs = D > 96 ? 2 : D > 64 ? 1 : 0;
  if (wide) return launch_bwd_wide(tm_q, tm_do, tm_k, tm_v, p, a, soft_cap, mask, stream);

  // dq (split form)
  p.out0 = static_cast<__nv_bfloat16*>(a.dq.data);
  p.out0_sb = a.dq.stride[0];
  p.out0_sh = a.dq.stride[1];
  p.out0_ss = a.dq.stride[2];
  p.out1 = nullptr;
  p.out1_sb = p.out1_sh = p.out1_ss = 0;
  p.row_ptr = a.sched_dq.row_ptr;
  p.entries = reinterpret_cast<const int4*>(a.sched_dq.entries);
  p.row_order = a.sched_dq.row_order;
  p.row_end = a.sched_dq.row_end;
  p.entries_per_batch = a.sched_dq.entries_per_batch;
  p.pmb = a.sched_dq.partial_mask_blocks;
  p.pm_bq = a.sched_dq.block_q > 0 ? a.sched_dq.block_q : kTile;
  p.pm_bkv = a.sched_dq.block_kv > 0 ? a.sched_dq.block_kv : kTile;
  p.n_rows = a.sched_dq.n_rows;
  // dq: the q heads of one kv head stream the same K / V
  p.n_groups = (int)(Hq * B);
  p.chunk_groups = chunk_groups_for(2 * Skv * kHeadDim * 2 / (Hq / Hkv), p.n_groups, Hq / Hkv);
  if ((int64_t)p.n_rows * p.n_groups > 0x7fffffffll) return SPLASH_ERR_TOO_LARGE;
  if (!fused && (mask & 2u))
    dq_kernel<<<dim3((unsigned)(p.n_rows * p.n_groups), 1u, 1u), kBwdThreads, kDqSmemBytes, stream>>>(
        tm_q, tm_do, tm_k, tm_v, p);
  if (cudaGetLastError() != cudaSuccess) return SPLASH_ERR_CUDA;

  // dkv
  p.out0 = static_cast<__nv_bfloat16*>(a.dk.data);
  p.out0_sb = a.dk.stride[0];
  p.out0_sh = a.dk.stride[1];
  p.out0_ss = a.dk.stride[2];
  p.out1 = static_cast<__nv_bfloat16*>(a.dv.data);
  p.out1_sb = a.dv.stride[0];
  p.out1_sh = a.dv.stride[1];
  p.out1_ss = a.dv.stride[2];
  p.out0_peer = a.dk_peer;
  p.out1_peer = a.dv_peer;
  p.row_ptr = a.sched_dkv.row_ptr;
  p.entries = reinterpret_cast<const int4*>(a.sched_dkv.entries);
  p.row_order = a.sched_dkv.row_order;
  p.row_end = a.sched_dkv.row_end;
  p.entries_per_batch = a.sched_dkv.entries_per_batch;
  p.pmb = a.sched_dkv.partial_mask_blocks;
  p.pm_bq = a.sched_dkv.block_q > 0 ? a.sched_dkv.block_q : kTile;
  p.pm_bkv = a.sched_dkv.block_kv > 0 ? a.sched_dkv.block_kv : kTile;
  p.n_rows = a.sched_dkv.n_rows;
  // dkv: the kv tiles of one (batch, kv head) stream the same Q / dO of its q-head group
  p.n_groups = (int)(Hkv * B);
  // (fused: plus the fp32 dQ image of those heads, which the reductions keep in L2)
  p.chunk_groups = chunk_groups_for((Hq / Hkv) * Sq * kHeadDim * (fused ? 8 : 4), p.n_groups, 1);
  p.main_groups = last_chunk(p.n_groups, p.chunk_groups, p.n_rows);
  if ((int64_t)p.n_rows * p.n_groups > 0x7fffffffll) return SPLASH_ERR_TOO_LARGE;
  if (mask & 4u) {
    const int64_t n_ctas = (int64_t)p.n_rows * p.n_groups;
    const int threads = fused ? kFusedThreads : kDkvThreads;
    p.n_split = dkv_split(a, shards, fused, nullptr);
    if (p.n_split < 0) return p.n_split;
    if (p.n_split > 1) dkv_kernel = dkv_kernel_for(true, fused, soft_cap, late);
    if (launch_clusters(dkv_kernel, (unsigned)n_ctas, p.n_split, threads, dkv_smem, stream, tm_q, tm_do, tm_k, tm_v, p) !=
        cudaSuccess)
      return SPLASH_ERR_CUDA;
  }
  if (fused && (mask & 2u)) {
    DqConvertParams cp;
    cp.acc = dq_acc;
    cp.dq = static_cast<__nv_bfloat16*>(a.dq.data);
    cp.dq_sb = a.dq.stride[0];
    cp.dq_sh = a.dq.stride[1];
    cp.dq_ss = a.dq.stride[2];
    cp.q_heads = (int)Hq;
    cp.n_q_tiles = (int)(Sq / kTile);
    cp.d_qk = (int)D;
    cp.scale = a.scale;
    cp.dq_peer = a.dq_peer;
    const int64_t n_tiles = B * Hq * (Sq / kTile);
    if (n_tiles > 0x7fffffffll) return SPLASH_ERR_TOO_LARGE;
    splash_dq_convert_kernel<<<(unsigned)n_tiles, 256, 0, stream>>>(cp);
  }
  return cudaGetLastError() == cudaSuccess ? SPLASH_OK : SPLASH_ERR_CUDA;
}

// ------------------------------------------------------------------------------------------
// backward with the scratch held in the library image (no allocation anywhere on the path)
// ------------------------------------------------------------------------------------------
// di rows followed by -logsumexp*log2(e) rows, SPLASH_STATIC_SCRATCH_MAX_ROWS each.
static __device__ __align__(256) float g_static_scratch[2 * SPLASH_STATIC_SCRATCH_MAX_ROWS];

int launch_bwd_static_scratch(const SplashBwdArgs& a, cudaStream_t stream) {
  const int64_t B = a.q.size[0], Hq = a.q.size[1], Sq = a.q.size[2];
  if (B <= 0 || Hq <= 0 || Sq <= 0) return SPLASH_ERR_INVALID_ARGUMENT;
  if (B * Hq * Sq > (int64_t)SPLASH_STATIC_SCRATCH_MAX_ROWS) return SPLASH_ERR_TOO_LARGE;

  // Inside host code the array's name is only a handle for the runtime, not a device address;
  // the address is looked up once per device, with that device current.
  constexpr int kMaxDevices = 64;
  static float* device_ptr[kMaxDevices] = {};
  static std::mutex mu;
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return SPLASH_ERR_CUDA;
  float* scratch = nullptr;
  {
    std::lock_guard<std::mutex> lock(mu);
    if (device_ptr[dev] == nullptr) {
      void* sym = nullptr;
      if (cudaGetSymbolAddress(&sym, g_static_scratch) != cudaSuccess || sym == nullptr) return SPLASH_ERR_CUDA;
      device_ptr[dev] = static_cast<float*>(sym);
    }
    scratch = device_ptr[dev];
  }
  SplashBwdArgs b = a;
  b.flags &= ~(uint32_t)SPLASH_BWD_FUSED_DQ;  // the array holds the two per-row terms only
  b.workspace = scratch;
  b.workspace_bytes = bwd_workspace_bytes(B, Hq, Sq);  // <= sizeof(g_static_scratch) by the row check
  return launch_bwd(b, SplashShards{}, stream);
}

}  // namespace sb
