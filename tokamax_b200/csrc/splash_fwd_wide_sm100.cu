// Splash attention forward for head dims above 128 (q / k up to 256 columns, v / o up to 256),
// bf16, sm_100a.  The reference's kernel test draws (256, 256) and (192, 128) among its head dims
// (splash_attention_kernel_test.py:233-237) and its microbenchmarks quote both; the kernel it
// replaces is `flash_attention_kernel` (splash_attention_kernel.py:299-527), as for the 128-wide
// forward.
//
// A CTA works on ONE 128-row q tile at a time (O alone takes up to 256 of the 512 TMEM columns) and streams K and V
// in tiles of 64 keys, as the backward at these head dims does (splash_bwd_wide_sm100.cu, which describes the
// layouts and the taking over of tiles):
//   TMEM  S of even steps 64 | S of odd steps 64 | O <= 256 | Q <= 128 (two bf16 a column)
//   smem  a ring of stages, each the V tile of a step n and the K tile of step n + 2; P of two steps.  Q goes through
//         the ring into TMEM, where it is the A operand of S = Q K^T (2 KB of shared memory read per MMA instead of
//         6).  P is an operand in shared memory, so that q k^T of step n + 2 need not wait for p v of step n
//   warps 0-3 / 4-7 softmax of the even / odd steps, warp 8 TMA producer and tile scheduler, warp 9 MMA
//         issuer (10, 11 idle: they complete the third warpgroup for the register hand-over)
// Once P(n) is there the issuer has everything for q k^T of step n + 2 and p v of step n, in that order: two waits
// and two commits a step.  The two warpgroups are at neighbouring steps at the same time.
//
// A row's maximum in use passes from step to step: a warpgroup takes the maximum of its 64 scores, waits for the
// maximum that the step before left in shared memory, raises it if it has to (by more than 2^8; O is then rescaled once
// p v of the step before has completed, a rare wait) and leaves it for the step behind, all ahead of its
// exponentials.  An even step that raises it looks at the odd step's scores too: the first maximum of a row is that of
// 128 keys, its largest weight 1 and not rounded, as in the 128-wide forward.  Each warpgroup sums its own steps' P,
// relative to the maximum it last saw; the two sums meet at the end.
// The schedule is the 128-wide forward's (rows = pairs of q tiles); a tile follows the entries in which it is live.
//
// What bounds it: the chain softmax -> q k^T -> softmax of a warpgroup's steps, 1400 cycles a step at (192, 128) and
// 1800 at 256 for 640 and 1024 of tensor time, and 6000 cycles between two tiles.  Before (steps of 128 keys, both
// warpgroups on one step, Q in shared memory, room for one step's K and V, a CTA a tile) -> this (us): causal 8192,
// 16 / 8 heads, head dim 256: 671 -> 431; causal 4096, 32 heads, (192, 128): 272 -> 203.  (The first step of a
// tile waits for the second one's scores: 5 us of each.  Raised by 64 keys alone, the maximum left the output 0.6 %
// further from its value in 64 bits.)  Measured beside it, without that wait: P over its
// scores in TMEM, rings of their own for K and V 441 / 209; the same with P in shared memory 475 / 206; that with q k^T
// and p v issued by two threads 454 / 196; this 429 / 195.
#include <mutex>

#include "splash_common.cuh"
#include "splash_fwd_params.cuh"

namespace sb {

constexpr int kWideFwdMaxSlots = 6;
constexpr int kWideFwdTileBytes = 7 * kTileBytes;       // P of two steps, both rings
constexpr int kWideFwdXchgBytes = 5 * kTile * 4;        // per row: maximum in use; a warpgroup's sum and largest score
constexpr int kWideFwdSmemBytes = kWideFwdTileBytes + kWideFwdXchgBytes + 512;

struct WideFwdBarriers {
  uint64_t answer[2];  // cluster launch control: what the request for the next tile returned
  int4 work[2];        // tiles in the order they are worked on: q tile (-1: none left), group, first live and last entry
  uint64_t answer_full;
  uint64_t work_full[2], work_empty[2];
  uint64_t q_ready;    // Q of a tile is in TMEM
  uint64_t full[kWideFwdMaxSlots], empty[kWideFwdMaxSlots];
  uint64_t s_full[2], p_full[2];  // per warpgroup, one phase per step of its own
  uint64_t o_done;     // a tile's O is complete,
  uint64_t o_free;     //   and has been read
  uint64_t m_full[4];  // per lane quarter, one phase per step: the step's maximum in use is in shared memory
  uint64_t x_full[4];  // per lane quarter, one phase per odd step: its scores' maximum is
  uint64_t l_full[4];  // per lane quarter, one phase per tile: both warpgroups' sums are
  uint32_t tmem_base;
  uint32_t abort_flag;
  uint32_t early_exit;
};
static_assert(sizeof(WideFwdBarriers) <= 512, "barrier block");

struct WideFwdParams {
  FwdParams f;
  int stages;
};

template <bool kSoftCap>
__global__ void __launch_bounds__(kFwdThreads, 1)
splash_fwd_wide_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                       const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ WideFwdParams wp) {
  constexpr uint32_t kColO = 2 * kSub, kColQ = 384;
  const FwdParams& p = wp.f;
  extern __shared__ __align__(1024) uint8_t smem[];
  const int halves_qk = (p.d_qk + 63) / 64, halves_v = (p.d_v + 63) / 64;  // 64-column halves of q / k, v / o
  const int bytes1 = halves_qk * kSubHalfBytes, bytes2 = halves_v * kSubHalfBytes;
  const uint32_t stages = (uint32_t)wp.stages;
  const int stage_bytes = bytes1 + bytes2;
  uint8_t* ring = smem + 2 * kHalfBytes;  // behind P: two tiles of 128 rows x 64 keys
  float* xchg = reinterpret_cast<float*>(smem + kWideFwdTileBytes);
  WideFwdBarriers* bars = reinterpret_cast<WideFwdBarriers*>(smem + kWideFwdTileBytes + kWideFwdXchgBytes);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    // (the swizzled tiles need a 1024-byte aligned base: a misaligned window is reported, not used)
    uint32_t bad = *reinterpret_cast<volatile uint32_t*>(p.err);
    if ((smem_u32(smem) & 1023u) != 0u) {
      if (atomicCAS(p.err, 0u, 2u) == 0u) {
        p.err[1] = blockIdx.x;
        p.err[2] = 0x2f20u;
        p.err[3] = smem_u32(smem);
      }
      bad = 2u;
    }
    bars->early_exit = bad;
    bars->abort_flag = 0;
    mbar_init(&bars->answer_full, 1);
    mbar_init(&bars->q_ready, 8);
    for (int i = 0; i < kWideFwdMaxSlots; ++i) {
      mbar_init(&bars->full[i], 1);
      mbar_init(&bars->empty[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&bars->work_full[i], 1);
      mbar_init(&bars->work_empty[i], 9);  // softmax warps and the MMA warp
      mbar_init(&bars->s_full[i], 1);
      mbar_init(&bars->p_full[i], 4);      // one arrival per warp of the warpgroup
    }
    for (int i = 0; i < 4; ++i) {
      mbar_init(&bars->m_full[i], 1);
      mbar_init(&bars->x_full[i], 1);
      mbar_init(&bars->l_full[i], 2);
    }
    mbar_init(&bars->o_done, 1);
    mbar_init(&bars->o_free, 8);
    mbar_fence_init();
  }
  __syncthreads();
  if (bars->early_exit != 0) return;  // an earlier CTA already reported a fault
  if (warp == 9) {
    tmem_alloc(&bars->tmem_base, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = bars->tmem_base;
  AbortCtx ab{&bars->abort_flag, p.err};

  RingPos work_pos{0, 0};
  auto next_work = [&](int4& w) {
    if (!mbar_wait(&bars->work_full[work_pos.slot], work_pos.phase, ab, 0x900u + work_pos.slot)) return false;
    w = bars->work[work_pos.slot];
    return true;
  };
  // state of a tile (of the schedule row's two) in an entry: 0 dead, 1 partial, 2 full
  auto state = [](const int4& ent, int tile) { return (ent.y >> (2 * (tile & 1))) & 3; };

  if (warp >= 8) {
   setmaxnreg_dec<kIssueRegs>();
   if (warp == 8) {
    // ------------------------------------------------------------------ TMA producer, tile scheduler
    if (elect_one()) {
      tma_prefetch_desc(&tm_q);
      tma_prefetch_desc(&tm_k);
      tma_prefetch_desc(&tm_v);
      RingPos pos{0, 0};
      uint32_t asked = 0;
      bool ok = true;
      int block = (int)blockIdx.x;
      while (ok) {
        int4 w = make_int4(-1, 0, 0, 0);
        const int4* entries = p.entries;
        if (block >= 0) {
          // two tiles per schedule row
          const CtaWork work = cta_work_at((unsigned)block >> 1, p.row_order, p.n_rows, p.n_groups, p.chunk_groups, true);
          const int batch = work.group / p.q_heads;
          entries += (int64_t)batch * p.entries_per_batch;
          w = make_int4(work.row * 2 + (block & 1), work.group, p.row_ptr[work.row],
                        p.row_end ? p.row_end[(int64_t)batch * p.n_rows + work.row] : p.row_ptr[work.row + 1]);
          while (w.z < w.w && state(entries[w.z], w.x) == 0) ++w.z;
          if (w.w < w.z) w.w = w.z;
        }
        if (block < 0 || w.x < p.n_q_tiles) {  // (odd number of q tiles: the last row has one)
          ok = mbar_wait(&bars->work_empty[work_pos.slot], work_pos.phase ^ 1u, ab, 0x910u + work_pos.slot);
          if (!ok) break;
          bars->work[work_pos.slot] = w;
          mbar_arrive(&bars->work_full[work_pos.slot]);
          work_pos.advance(1, 2);
          if (block < 0) break;
          const int head = w.y % p.q_heads, batch = w.y / p.q_heads;
          const int kv_head = head / (p.q_heads / p.kv_heads);
          // One stage: a 64-row tile of Q or K in front (row1 < 0: none), one of V behind it (row2 < 0: none).  A tile's
          // stages: Q, Q, K(0), K(1), then V(n) with K(n + 2).
          auto load = [&](const CUtensorMap* tm, int row1, int head1, int row2) {
            if (!mbar_wait(&bars->empty[pos.slot], pos.phase ^ 1u, ab, 0x800u + pos.slot)) return false;
            uint8_t* dst = ring + pos.slot * stage_bytes;
            mbar_arrive_expect_tx(&bars->full[pos.slot], (uint32_t)((row1 >= 0 ? bytes1 : 0) + (row2 >= 0 ? bytes2 : 0)));
            if (row1 >= 0)
              for (int i = 0; i < halves_qk; ++i)
                tma_load_4d(dst + i * kSubHalfBytes, tm, &bars->full[pos.slot], i * 64, row1, head1, batch);
            if (row2 >= 0)
              for (int i = 0; i < halves_v; ++i)
                tma_load_4d(dst + bytes1 + i * kSubHalfBytes, &tm_v, &bars->full[pos.slot], i * 64, row2, kv_head, batch);
            pos.advance(1, stages);
            return true;
          };
          if (w.z < w.w) {
            for (int sub = 0; sub < 2 && ok; ++sub) ok = load(&tm_q, w.x * kTile + sub * kSub, head, -1);
            int v_row = entries[w.z].x * kTile;
            for (int sub = 0; sub < 2 && ok; ++sub) ok = load(&tm_k, v_row + sub * kSub, kv_head, -1);
            for (int e = w.z + 1; e <= w.w && ok; ++e) {
              int k_row = -1;
              if (e < w.w) {
                const int4 ent = entries[e];
                if (state(ent, w.x) == 0) continue;
                k_row = ent.x * kTile;
              }
              for (int sub = 0; sub < 2 && ok; ++sub) ok = load(&tm_k, k_row < 0 ? -1 : k_row + sub * kSub, kv_head, v_row + sub * kSub);
              v_row = k_row;
            }
          }
          if (!ok) break;
        }
        // the next tile: asked for when all of this one is on its way, and no earlier (see the backward)
        mbar_arrive_expect_tx(&bars->answer_full, 16);
        clc_request(bars->answer, &bars->answer_full);
        ok = mbar_wait(&bars->answer_full, asked & 1u, ab, 0x920u);
        ++asked;
        if (ok) block = clc_block(bars->answer);
        fence_proxy_async_smem();  // read before the next answer overwrites it
      }
    }
   } else if (warp == 9) {
    // ------------------------------------------------------------------ MMA issuer
    if (elect_one()) {
      constexpr uint32_t idesc_qk = make_idesc_bf16(kTile, kSub, false, false);
      const uint32_t idesc_pv = make_idesc_bf16(kTile, halves_v * 64, false, true);
      const uint32_t ring_addr = smem_u32(ring);
      RingPos pos{0, 0};
      uint32_t stepped = 0;  // tiles with steps so far
      bool ok = true;
      // S(n) = Q K^T: A in TMEM, K = 16 a slice, four slices a 64-column half
      auto issue_qk = [&](uint32_t n) {
        const uint32_t d = tmem + (n & 1u) * kSub;
        const SmemDesc db = make_smem_desc_sw128(ring_addr + pos.slot * stage_bytes, 16, 1024);
        auto slice = [&](int h, int k) {
          umma_ts(d, tmem + kColQ + h * 32 + k * 8, desc_at(db, h * kSubHalfBytes + k * 32), idesc_qk, (h + k) > 0 ? 1u : 0u);
        };
#pragma unroll
        for (int h = 0; h < 4; ++h) {
          if (4 * h >= p.nk_qk) break;
          if (4 * h + 4 <= p.nk_qk) {
#pragma unroll
            for (int k = 0; k < 4; ++k) slice(h, k);
          } else {
            for (int k = 0; 4 * h + k < p.nk_qk; ++k) slice(h, k);
          }
        }
        tc_commit(&bars->s_full[n & 1u]);
      };
      auto wait_stage = [&]() { return mbar_wait(&bars->full[pos.slot], pos.phase, ab, 0xA10u + pos.slot); };
      auto release_stage = [&]() {
        tc_commit(&bars->empty[pos.slot]);
        pos.advance(1, stages);
      };
      uint32_t ph = 0;
      for (;;) {
        int4 w;
        if (!next_work(w)) break;
        mbar_arrive(&bars->work_empty[work_pos.slot]);
        work_pos.advance(1, 2);
        if (w.x < 0) break;
        if (w.z >= w.w) continue;
        const int4* entries = p.entries + (int64_t)(w.y / p.q_heads) * p.entries_per_batch;
        ok = mbar_wait(&bars->q_ready, stepped & 1u, ab, 0xA00u);
        if (!ok) break;
        for (int i = 0; i < 2; ++i) {  // Q's two stages are free again
          mbar_arrive(&bars->empty[pos.slot]);
          pos.advance(1, stages);
        }
        for (uint32_t n = 0; n < 2 && ok; ++n) {
          ok = wait_stage();
          if (!ok) break;
          mma_issue_fence();
          issue_qk(n);
          release_stage();
        }
        if (ok && stepped > 0) ok = mbar_wait(&bars->o_free, (stepped - 1) & 1u, ab, 0xA50u);
        bool acc = false;
        int e = w.z;
        while (e < w.w && ok) {  // a live entry: two steps
          int ahead = e + 1;
          int4 ent = make_int4(0, 0, 0, 0);
          if (ahead < w.w) ent = entries[ahead];
          while (ahead < w.w && state(ent, w.x) == 0)
            if (++ahead < w.w) ent = entries[ahead];
          for (uint32_t sub = 0; sub < 2 && ok; ++sub) {
            ok = wait_stage() && mbar_wait(&bars->p_full[sub], ph, ab, 0xA30u + sub);
            if (!ok) break;
            mma_issue_fence();
            if (ahead < w.w) issue_qk(sub);
            // O (+)= P V: P K-major, V read MN-major, K = 64 keys in four slices
            const SmemDesc da = make_smem_desc_sw128(smem_u32(smem) + sub * kHalfBytes, 16, 1024);
            const SmemDesc db = make_smem_desc_sw128(ring_addr + pos.slot * stage_bytes + bytes1, kSubHalfBytes, 1024);
#pragma unroll
            for (int k = 0; k < 4; ++k)
              umma_ss(tmem + kColO, desc_at(da, k * 32), desc_at(db, k * 2048), idesc_pv, (acc || k > 0) ? 1u : 0u);
            acc = true;
            release_stage();
          }
          ph ^= 1u;
          e = ahead;
        }
        if (!ok) break;
        tc_commit(&bars->o_done);
        ++stepped;
      }
    }
   }
  } else {
    // ------------------------------------------------------------------ softmax warpgroups
    setmaxnreg_inc<kSoftmaxRegs>();
    const int set = warp >> 2;         // steps n % 2 = set
    const int wq = warp & 3;           // TMEM lane quarter this warp may touch
    const int r = wq * 32 + lane;      // row within the tile
    const uint32_t lane_addr = (uint32_t)(wq * 32) << 16;
    const uint32_t t_s = tmem + lane_addr + set * kSub;
    const uint32_t t_o = tmem + lane_addr + kColO;
    const bool has_seg = p.q_seg != nullptr;
    const bool fixed_max = p.max_logit_value != nullptr;
    const float c = fmaxf(kSoftCap ? p.soft_cap * kLog2e : p.scale_log2, kMinScaleLog2);  // score -> log2 units
    // 32-column groups of O that hold real columns, shared out between the two warpgroups
    const int o_groups = (p.d_v + 31) / 32;
    const int og_begin = set == 0 ? 0 : (o_groups + 1) / 2;
    const int og_end = set == 0 ? (o_groups + 1) / 2 : o_groups;
    uint8_t* p_row = smem + set * kHalfBytes + r * 128;  // this row of this warpgroup's P
    float* m_row = xchg + r;                     // the row's maximum in use, as the last step left it
    float* l_row = xchg + kTile + r;             // [warpgroup]: its share of the row's sum
    float* true_row = xchg + 3 * kTile + r;      // [warpgroup]: the largest score it saw
    float* x_row = true_row + kTile;             // until then: the maximum of an odd step's scores
    RingPos base{0, 0};     // stage at which the next tile begins
    uint32_t ph = 0;        // parity of this warpgroup's steps
    uint32_t stepped = 0;   // tiles with steps so far

    // takes the next tile and carries its Q to TMEM: row r of the tile in lane r, 64 head-dim columns at a time, the
    // warpgroups in turn (every q k^T of the last tile has completed)
    auto take_work = [&](int4& w) {
      bool ok = next_work(w);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) return false;
      if (lane == 0) mbar_arrive(&bars->work_empty[work_pos.slot]);
      work_pos.advance(1, 2);
      if (w.x < 0 || w.z >= w.w) return true;
      RingPos pos = base;
      if (wq >= 2) pos.advance(1, stages);
      ok = mbar_wait(&bars->full[pos.slot], pos.phase, ab, 0xB40u + pos.slot);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) return false;
      for (int h = set; h < halves_qk; h += 2) {
        const uint8_t* src = ring + pos.slot * stage_bytes + h * kSubHalfBytes + (r & 63) * 128;
        uint32_t v[32];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const uint4 x = *reinterpret_cast<const uint4*>(src + ((j ^ (r & 7)) << 4));
          v[4 * j] = x.x, v[4 * j + 1] = x.y, v[4 * j + 2] = x.z, v[4 * j + 3] = x.w;
        }
        tmem_st32(tmem + lane_addr + kColQ + h * 32, v);
      }
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bars->q_ready);
      return true;
    };

    int4 cur;
    bool ok = take_work(cur);
    while (ok && cur.x >= 0) {
      const int tile = cur.x, head = cur.y % p.q_heads, batch = cur.y / p.q_heads, eend = cur.w;
      const int4* entries = p.entries + (int64_t)batch * p.entries_per_batch;
      const int q_row = tile * kTile + r;
      const int qi = p.q_sequence ? p.q_sequence[q_row] : q_row;
      const RowInterval iv = mask_fn_interval(p.fn, qi);
      const int q_seg = has_seg ? p.q_seg[(int64_t)batch * p.q_len + q_row] : 0;
      const int32_t* kv_seg_row = has_seg ? p.kv_seg + (int64_t)batch * p.kv_len : nullptr;

      float m_used = -INFINITY;  // scaled (log2) units
      float m_true = kMaskedLogit;
      float l = 0.f;             // this warpgroup's share of the row sum (a sink is counted by the first)
      float sink2 = -INFINITY;   // sink logit in log2 units
      if (p.sinks != nullptr) sink2 = p.sinks[head] * kLog2e;
      if (fixed_max) {
        m_used = p.max_logit_value[head] * kLog2e;
        if (p.sinks != nullptr && set == 0) l = ex2(sink2 - m_used);
      } else if (p.sinks != nullptr) {
        m_used = sink2;
        if (set == 0) l = 1.f;
      }
      uint32_t live_entries = 0;
      // stage of p v of this warpgroup's last step, whose release says that those MMAs have completed
      RingPos last = base;
      last.skip(2 + set, stages);  // (two ahead of its first step's, that tile's fifth or sixth)

      int4 ent_next = cur.z < eend ? entries[cur.z] : make_int4(0, 0, 0, 0);
      for (int e = cur.z; e < eend; ++e) {
        const int4 ent = ent_next;
        if (e + 1 < eend) ent_next = entries[e + 1];
        const int st = state(ent, tile);
        if (st == 0) continue;
        const bool first = live_entries++ == 0 && set == 0;  // step 0
        ok = mbar_wait(&bars->s_full[set], ph, ab, 0xB00u + set);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        tc_fence_after();

        float s[kSub];
        {
          uint32_t v0[32], v1[32];
          tmem_ld32(t_s, v0);
          tmem_ld32(t_s + 32, v1);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 32; ++j) {
            s[j] = __uint_as_float(v0[j]);
            s[32 + j] = __uint_as_float(v1[j]);
          }
        }
        if constexpr (kSoftCap) {
          tanh_all(s, p.softcap_a);
        }
        const int kv0 = ent.x * kTile + set * kSub;  // first key of this step
        if (st == 1) {
          if (p.fn.kind != SPLASH_MASK_TABLE) {
            const int lo_rel = iv.lo <= kv0 ? 0 : iv.lo - kv0;
            const int hi_rel = iv.hi >= kv0 + (kSub - 1) ? kSub - 1 : iv.hi - kv0;
#pragma unroll
            for (int j = 0; j < kSub; ++j)
              if (j < lo_rel || j > hi_rel) s[j] = kMaskedLogit;
          } else {
            const int pid = (tile & 1) == 0 ? ent.z : ent.w;
            const int8_t* mrow = p.pmb + ((int64_t)pid * p.pm_bq + (q_row % p.pm_bq)) * p.pm_bkv + (kv0 % p.pm_bkv);
            const int4* m4 = reinterpret_cast<const int4*>(mrow);
#pragma unroll
            for (int g = 0; g < kSub / 16; ++g) {
              const int4 mv = __ldg(m4 + g);
              const uint32_t w[4] = {(uint32_t)mv.x, (uint32_t)mv.y, (uint32_t)mv.z, (uint32_t)mv.w};
#pragma unroll
              for (int j = 0; j < 16; ++j)
                if (((w[j >> 2] >> ((j & 3) * 8)) & 0xffu) == 0u) s[g * 16 + j] = kMaskedLogit;
            }
          }
        }
        if (has_seg && !((ent.y >> (4 + (tile & 1))) & 1)) {  // (bit set: the whole tile lies inside one segment)
          const int4* sg4 = reinterpret_cast<const int4*>(kv_seg_row + kv0);
#pragma unroll
          for (int g = 0; g < kSub / 4; ++g) {
            const int4 sv = __ldg(sg4 + g);
            if (sv.x != q_seg) s[g * 4 + 0] = kMaskedLogit;
            if (sv.y != q_seg) s[g * 4 + 1] = kMaskedLogit;
            if (sv.z != q_seg) s[g * 4 + 2] = kMaskedLogit;
            if (sv.w != q_seg) s[g * 4 + 3] = kMaskedLogit;
          }
        }

        float mx0 = max3(s[0], s[1], s[2]), mx1 = max3(s[3], s[4], s[5]);
        float mx2 = max3(s[6], s[7], s[8]), mx3 = max3(s[9], s[10], s[11]);
#pragma unroll
        for (int j = 12; j < kSub - 4; j += 8) {
          mx0 = max3(mx0, s[j], s[j + 1]);
          mx1 = max3(mx1, s[j + 2], s[j + 3]);
          mx2 = max3(mx2, s[j + 4], s[j + 5]);
          mx3 = max3(mx3, s[j + 6], s[j + 7]);
        }
        mx0 = max3(mx0, s[kSub - 4], s[kSub - 3]);
        mx1 = max3(mx1, s[kSub - 2], s[kSub - 1]);
        const float mx = fmaxf(fmaxf(mx0, mx1), fmaxf(mx2, mx3));
        m_true = fmaxf(m_true, mx);
        if (!fixed_max) {
          float m_new = fmaxf(mx * c, kLogitFloor);
          if (set == 1) {
            *x_row = m_new;
            __syncwarp();
            if (lane == 0) mbar_arrive(&bars->x_full[wq]);
          }
          // the maximum in use of the step before (the steps of a tile are an even number: phase n of the barrier has
          // parity n & 1, and step n belongs to warpgroup n & 1)
          float m_in = m_used;
          if (!first) {
            ok = mbar_wait(&bars->m_full[wq], (uint32_t)(set ^ 1), ab, 0xB30u);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            m_in = *m_row;
          }
          const bool raise = __any_sync(0xffffffffu, m_new > m_in + kRescaleThreshold);
          float m_next = m_in;
          if (raise) {
            if (set == 0) {
              // (an odd step leaves its scores' maximum, then waits for the even one's m_full: neither the phase before
              // this one nor the one behind it can be in progress)
              ok = mbar_wait(&bars->x_full[wq], ph, ab, 0xB80u);
              ok = __all_sync(0xffffffffu, ok);
              if (!ok) break;
              m_new = fmaxf(m_new, *x_row);
            }
            m_next = fmaxf(m_in, m_new);
          }
          *m_row = m_next;
          __syncwarp();
          if (lane == 0) mbar_arrive(&bars->m_full[wq]);
          if (m_next != m_used) l *= ex2(m_used - m_next);
          m_used = m_next;
          if (raise && !first) {
            // O still receives p v of the step before, the other warpgroup's: wait for it before touching O
            RingPos other = last;
            other.advance(1, stages);
            ok = mbar_wait(&bars->empty[other.slot], other.phase, ab, 0xB10u);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            tc_fence_after();
            const float alpha = m_in != m_next ? ex2(m_in - m_next) : 1.f;
            for (int g = 0; g < o_groups; ++g) {
              uint32_t v[32];
              tmem_ld32(t_o + g * 32, v);
              tmem_ld_wait();
#pragma unroll
              for (int j = 0; j < 32; ++j) v[j] = __float_as_uint(__uint_as_float(v[j]) * alpha);
              tmem_st32(t_o + g * 32, v);
            }
          }
        }

        if (live_entries > 1) {  // P of this warpgroup's last step has been multiplied: its tile is free
          ok = mbar_wait(&bars->empty[last.slot], last.phase, ab, 0xB70u + set);
          ok = __all_sync(0xffffffffu, ok);
          if (!ok) break;
        }
        last.advance(2, stages);
        const float2 c2 = make_float2(c, c), nm2 = make_float2(-m_used, -m_used);
        float2 lsa = make_float2(0.f, 0.f), lsb = make_float2(0.f, 0.f);
#pragma unroll
        for (int ch = 0; ch < 8; ++ch) {  // eight keys: a 16-byte chunk of the row's 128 bytes, at ch ^ (row mod 8)
          uint32_t pk[4];
#pragma unroll
          for (int j = 0; j < 4; j += 2) {
            const float2 xa = __ffma2_rn(make_float2(s[ch * 8 + 2 * j], s[ch * 8 + 2 * j + 1]), c2, nm2);
            const float2 xb = __ffma2_rn(make_float2(s[ch * 8 + 2 * j + 2], s[ch * 8 + 2 * j + 3]), c2, nm2);
            const float2 pa = make_float2(ex2(xa.x), ex2(xa.y));
            const float2 pb = make_float2(ex2(xb.x), ex2(xb.y));
            lsa = __fadd2_rn(lsa, pa);
            lsb = __fadd2_rn(lsb, pb);
            pk[j] = pack_bf16(pa.x, pa.y);
            pk[j + 1] = pack_bf16(pb.x, pb.y);
          }
          *reinterpret_cast<uint4*>(p_row + ((ch ^ (r & 7)) << 4)) = make_uint4(pk[0], pk[1], pk[2], pk[3]);
        }
        l += (lsa.x + lsb.x) + (lsa.y + lsb.y);
        fence_proxy_async_smem();  // generic-proxy stores -> visible to the MMA's async-proxy reads
        tmem_st_wait();            // (a rescaled O)
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&bars->p_full[set]);
        ph ^= 1u;
      }
      if (!ok) break;

      const bool steps = live_entries > 0;
      float m_all = m_used, l_all = l, true_all = m_true;
      if (steps) {
        // the sums of the two warpgroups meet, relative to the maximum that the last step left
        if (!fixed_max && set == 0) {
          ok = mbar_wait(&bars->m_full[wq], 1u, ab, 0xB60u);
          ok = __all_sync(0xffffffffu, ok);
          if (!ok) break;
          m_all = *m_row;
        }
        l_row[set * kTile] = m_used == m_all ? l : l * ex2(m_used - m_all);  // (also where the maximum is infinite)
        true_row[set * kTile] = m_true;
        __syncwarp();
        if (lane == 0) mbar_arrive(&bars->l_full[wq]);
        ok = mbar_wait(&bars->l_full[wq], stepped & 1u, ab, 0xB50u);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        l_all = l_row[0] + l_row[kTile];
        true_all = fmaxf(true_row[0], true_row[kTile]);
        ok = mbar_wait(&bars->o_done, stepped & 1u, ab, 0xB20u);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        tc_fence_after();
        base.skip(4 + 2 * live_entries, stages);
        ++stepped;
      }
      // The next tile's scores can start before this tile's rows are stored.
      int4 next;
      ok = take_work(next);
      if (!ok) break;
      // ---- O / l -> bf16 (each warpgroup its share of the columns), logsumexp, max_logits
      const bool live = l_all > 0.f;  // a row that met a live key, or has a sink
      const float inv = live ? 1.0f / l_all : 0.f;
      __nv_bfloat16* row0 = p.o + (int64_t)batch * p.o_sb + (int64_t)head * p.o_sh + (int64_t)(tile * kTile + wq * 32) * p.o_ss;
      for (int g = og_begin; g < og_end; ++g) {
        uint32_t v[32];
#pragma unroll
        for (int j = 0; j < 32; ++j) v[j] = 0u;
        if (steps) {
          tmem_ld32(t_o + g * 32, v);
          tmem_ld_wait();
        }
        store_rows32(row0, p.o_ss, v, inv, g * 32, p.d_v);
      }
      if (steps) {
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&bars->o_free);
      }
      if (set == 0) {
        const int64_t stat = ((int64_t)batch * p.q_heads + head) * p.q_len + q_row;
        if (p.lse) p.lse[stat] = live ? (m_all + log2f(l_all)) * kLn2 : p.mask_value;
        if (p.maxl) {
          float mv = true_all * (kSoftCap ? p.soft_cap : p.scale);
          if (p.sinks != nullptr) mv = fmaxf(mv, sink2 * kLn2);
          if (fixed_max) mv = m_all * kLn2;
          p.maxl[stat] = live ? mv : p.mask_value;
        }
      }
      cur = next;
    }
  }

  // ---- teardown
  tc_fence_before();
  __syncthreads();
  if (warp == 9) {
    __syncwarp();
    drain_after_give_up(&bars->abort_flag);
    tmem_dealloc(tmem, 512);
  }
}

int launch_fwd_wide(const CUtensorMap& tm_q, const CUtensorMap& tm_k, const CUtensorMap& tm_v,
                    const FwdParams& p, bool soft_cap, cudaStream_t stream) {
  const int64_t blocks = 2ll * p.n_rows * p.n_groups;
  if (blocks > 0x7fffffffll) return SPLASH_ERR_TOO_LARGE;
  auto* kernel = soft_cap ? splash_fwd_wide_kernel<true> : splash_fwd_wide_kernel<false>;
  {
    static std::mutex attr_mu;
    static bool attr_done[64][2] = {};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return SPLASH_ERR_CUDA;
    std::lock_guard<std::mutex> lock(attr_mu);
    if (!attr_done[dev][soft_cap ? 1 : 0]) {
      if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kWideFwdSmemBytes) != cudaSuccess)
        return SPLASH_ERR_CUDA;
      attr_done[dev][soft_cap ? 1 : 0] = true;
    }
  }
  WideFwdParams wp;
  wp.f = p;
  const int stage_bytes = ((p.d_qk + 63) / 64 + (p.d_v + 63) / 64) * kSubHalfBytes;
  wp.stages = (kWideFwdTileBytes - 2 * kHalfBytes) / stage_bytes;  // three and more
  if (wp.stages > kWideFwdMaxSlots) wp.stages = kWideFwdMaxSlots;
  kernel<<<(unsigned)blocks, kFwdThreads, kWideFwdSmemBytes, stream>>>(tm_q, tm_k, tm_v, wp);
  return cudaGetLastError() == cudaSuccess ? SPLASH_OK : SPLASH_ERR_CUDA;
}

}  // namespace sb
