// Splash attention backward for head dims above 128 (q / k up to 256 columns, v / o up to 256),
// bf16, sm_100a: dq, dk and dv as passes of one kernel.  Same arithmetic as the 128-wide
// backward (reference: splash_attention_kernel.py:1234-1459, base.py:115-173): P = exp(S - lse),
// dS = P * (dP - di), dq = dS k, dk = dS^T q, dv = P^T do, the q heads of a kv head summed inside
// one CTA (no atomics, bitwise repeatable).
//
// A CTA keeps one 128-row tile (the stationary side) and streams the other side in tiles of 64 rows, so that
// scores are 128 x 64: that is what leaves room in TMEM and shared memory for the next step's scores and
// operands beside this step's, and the tensor core works on one step while the element-wise warps are at another.
//
// pass   stationary          streamed, 64 rows a step    output                       taken when
//  dq    Q (TMEM), dO        K (held), V                 dq += dS k                   always
//  dkv   K, V                Q, dO (both held)           dk += dS^T q, dv += P^T do   both outputs fit TMEM (320 columns)
//  dk    K (TMEM), V         Q (held), dO                dk += dS^T q                 otherwise
//  dv    K (TMEM)            Q, dO (held)                dv += P^T do                 otherwise
//
// "Held" tiles feed an output MMA as its MN-major B operand and stay until that has completed; the others
// go when the scores are done.  Where the table says TMEM, the stationary operand of the scores is copied
// there once, as the MMA's A operand: S = A B^T then reads 2 KB of shared memory per MMA instead of 6 KB and the
// operand takes none.  Every streamed tile lies as 64-column halves of 64 rows x 128 bytes (128-byte swizzle).
//
// TMEM (512 columns)   dq, dk:  S 64 | S 64 | dP 64 | output <= 192 | A <= 96     packed dS over its S columns
//       d_qk > 192:             S 64 | dP 64 | output 256 | A 128                 packed dS over the dP columns
//                      dv:      S 64 | S 64 | output <= 256 | A <= 128            packed P over its S columns
//                      dkv:     S 64 | S 64 | dP 64 | dk, dv <= 320               packed P and dS over their S columns
//
// Sixteen compute warps in two sets of eight: a set takes every second step, 32 of its 64 columns a thread.
// While one set waits for dP or writes dS, the other is at the exponentials of the next step.
// In the dk / dv passes the tile is transposed (threads own kv rows, columns are query rows): logsumexp and di
// come per column, brought into shared memory with the held tile.
//
// CTAs stay for several tiles: the producer takes over CTAs that have not been launched yet (cluster launch
// control), posts their tiles and goes on loading, so that a tile's outputs are stored, and its successor's
// operands loaded, beside MMAs.  One tile a CTA spent 20,000 of 75,000 cycles between two loops.
//
// What bounds it: the shared-memory pipe (operand reads of the 128 x 64 score MMAs, the streamed tiles coming in,
// statistics) together with the tensor core, at 1500 (dq), 1950 (dkv) cycles a step for (192, 128), 2150 (dq), 2250
// (dk), 1300 (dv) for 256.  Measured, three passes over 128 x 128 tiles that a CTA each computed one after the
// other -> this (us, a pause before each pass): causal 4096, 32 heads, (192, 128): dq 403 -> 244, dk and dv 727 -> 323;
// causal 8192, 16 / 8 heads, head dim 256: dq 781 -> 636, dk 925 -> 649, dv 603 -> 399.
#include <mutex>

#include "splash_common.cuh"
#include "splash_bwd_params.cuh"

namespace sb {

enum WidePass { kWideDq = 0, kWideDkv = 1, kWideDk = 2, kWideDv = 3 };

constexpr int kWideThreads = 576;  // 16 compute warps, TMA warp, MMA warp
constexpr int kWideTmaWarp = 16;
constexpr int kWideMmaWarp = 17;
constexpr int kWideMaxSlots = 4;
constexpr int kWideTileBytes = 7 * kTileBytes;  // operand tiles
constexpr int kWideStatsBytes = kWideMaxSlots * 2 * kSub * 4;  // a slot: -lse log2(e), -di of its query rows
constexpr int kWideSmemBytes = kWideTileBytes + kWideStatsBytes + 512;
constexpr int kWideBothColumns = 512 - 3 * kSub;  // dk and dv columns that one pass can hold

struct WideParams {
  BwdParams b;
  int n1, n2;               // slots of the rings of the streamed operand of S, and of dP / of the dv MMA
};

struct WideBwdBarriers {
  uint64_t answer[2];    // cluster launch control: what the request for the next tile returned
  int4 work[2];          // tiles in the order they are worked on: tile (-1: none left), group, first and last entry
  uint64_t answer_full;
  uint64_t work_full[2], work_empty[2];
  uint64_t a1_ready;     // stationary operands of a tile: of the scores (in TMEM, or its TMA has landed),
  uint64_t a2_full;      //   of dP,
  uint64_t stat_free;    //   and the last MMA that reads them has completed
  uint64_t full1[kWideMaxSlots], empty1[kWideMaxSlots];
  uint64_t full2[kWideMaxSlots], empty2[kWideMaxSlots];
  // per set of compute warps (steps n with n % 2 = set)
  uint64_t s_full[2];
  uint64_t s_free[2];    // one S buffer: the set has read its scores
  uint64_t dp_full[2];
  uint64_t p_full[2];    // dkv / dv: packed P in TMEM
  uint64_t ds_full[2];   // packed dS in TMEM, dP read
  uint64_t acc_done;     // a tile's outputs are complete,
  uint64_t out_free;     //   and have been read
  uint32_t tmem_base;
  uint32_t abort_flag;
  uint32_t early_exit;
};
static_assert(sizeof(WideBwdBarriers) <= 512, "barrier block");

// kOneS (dq, dk): one S buffer, for head dims whose output and stationary operand leave no columns for a second.
template <int kPass, bool kSoftCap, bool kOneS>
__global__ void __launch_bounds__(kWideThreads, 1)
splash_bwd_wide_kernel(const __grid_constant__ CUtensorMap tm_a1, const __grid_constant__ CUtensorMap tm_a2,
                       const __grid_constant__ CUtensorMap tm_x1, const __grid_constant__ CUtensorMap tm_x2,
                       const __grid_constant__ WideParams wp) {
  constexpr bool kHasDp = kPass != kWideDv;
  constexpr bool kHasP = kPass == kWideDkv || kPass == kWideDv;   // P feeds an MMA
  constexpr bool kA1Tmem = kPass != kWideDkv;
  static_assert(!kOneS || kPass == kWideDq || kPass == kWideDk, "");
  // packed P: over the first 16 of the 32 score columns that a thread reads; packed dS: behind it (dkv), in its
  // place (dq, dk), or over the dP columns (one S buffer: the scores' columns are the next step's by then)
  constexpr uint32_t kColDp = kOneS ? kSub : 2 * kSub;
  constexpr uint32_t kColOut = kColDp + (kHasDp ? kSub : 0);
  constexpr uint32_t kColA1 = 384;
  constexpr uint32_t kDsOffset = kPass == kWideDkv ? 16 : 0;
  const BwdParams& p = wp.b;

  extern __shared__ __align__(1024) uint8_t smem[];
  const int halves_qk = (p.d_qk + 63) / 64, halves_v = (p.d_v + 63) / 64;  // 64-column halves of q / k, v / do
  uint8_t* a1_smem = smem;
  uint8_t* a2_smem = a1_smem + (kA1Tmem ? 0 : halves_qk * kHalfBytes);
  uint8_t* ring1 = a2_smem + (kHasDp ? halves_v * kHalfBytes : 0);
  uint8_t* ring2 = ring1 + wp.n1 * halves_qk * kSubHalfBytes;
  float* stats = reinterpret_cast<float*>(smem + kWideTileBytes);
  WideBwdBarriers* bars = reinterpret_cast<WideBwdBarriers*>(smem + kWideTileBytes + kWideStatsBytes);
  const uint32_t n1 = (uint32_t)wp.n1, n2 = (uint32_t)wp.n2;
  const int bytes1 = halves_qk * kSubHalfBytes, bytes2 = halves_v * kSubHalfBytes;

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int group = p.q_heads / p.kv_heads;
  // dq pass: a tile belongs to one (batch, q head); the others: to one (batch, kv head) and walk its q heads
  const int heads_here = kPass == kWideDq ? 1 : group;
  const int n_own = kPass == kWideDq ? p.q_heads : p.kv_heads;

  if (threadIdx.x == 0) {
    // The swizzled tiles need a 1024-byte aligned base; there is no slack in the allocation to fix it
    // up, so a misaligned window is reported, not used.
    uint32_t bad = *reinterpret_cast<volatile uint32_t*>(p.err);
    if ((smem_u32(smem) & 1023u) != 0u) {
      if (atomicCAS(p.err, 0u, 2u) == 0u) {
        p.err[1] = blockIdx.x;
        p.err[2] = 0x2f10u;
        p.err[3] = smem_u32(smem);
      }
      bad = 2u;
    }
    bars->early_exit = bad;
    bars->abort_flag = 0;
    mbar_init(&bars->answer_full, 1);
    mbar_init(&bars->a1_ready, kA1Tmem ? 16 : 1);
    mbar_init(&bars->a2_full, 1);
    mbar_init(&bars->stat_free, 1);
    for (int i = 0; i < kWideMaxSlots; ++i) {
      mbar_init(&bars->full1[i], 1);
      mbar_init(&bars->empty1[i], 1);
      mbar_init(&bars->full2[i], 1);
      mbar_init(&bars->empty2[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&bars->work_full[i], 1);
      mbar_init(&bars->work_empty[i], 17);  // compute warps and the MMA warp
      mbar_init(&bars->s_full[i], 1);
      mbar_init(&bars->s_free[i], 8);       // one arrival per warp of the set
      mbar_init(&bars->dp_full[i], 1);
      mbar_init(&bars->p_full[i], 8);
      mbar_init(&bars->ds_full[i], 8);
    }
    mbar_init(&bars->acc_done, 1);
    mbar_init(&bars->out_free, 16);
    mbar_fence_init();
  }
  __syncthreads();
  if (bars->early_exit != 0) return;
  if (warp == kWideMmaWarp) {
    tmem_alloc(&bars->tmem_base, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = bars->tmem_base;
  AbortCtx ab{&bars->abort_flag, p.err};

  // The tile that comes next, as the producer posted it.
  RingPos work_pos{0, 0};
  auto next_work = [&](int4& w) {
    if (!mbar_wait(&bars->work_full[work_pos.slot], work_pos.phase, ab, 0xB00u + work_pos.slot)) return false;
    w = bars->work[work_pos.slot];
    return true;
  };
  auto work_read = [&]() {  // one thread of each warp that called next_work
    mbar_arrive(&bars->work_empty[work_pos.slot]);
  };

  if (warp == kWideTmaWarp) {
    // ------------------------------------------------------------------ TMA producer, tile scheduler
    if (elect_one()) {
      tma_prefetch_desc(&tm_a1);
      tma_prefetch_desc(&tm_a2);
      tma_prefetch_desc(&tm_x1);
      tma_prefetch_desc(&tm_x2);
      RingPos r1{0, 0}, r2{0, 0};
      uint32_t stepped = 0;  // tiles with steps so far
      uint32_t asked = 0;
      bool ok = true;
      int block = (int)blockIdx.x;
      while (ok) {
        // post the tile
        int4 w = make_int4(-1, 0, 0, 0);
        if (block >= 0) {
          const CtaWork work = cta_work_at((unsigned)block, p.row_order, p.n_rows, p.n_groups, p.chunk_groups, true);
          const int batch = work.group / n_own;
          w = make_int4(work.row, work.group, p.row_ptr[work.row],
                        p.row_end ? p.row_end[(int64_t)batch * p.n_rows + work.row] : p.row_ptr[work.row + 1]);
          if (w.w < w.z) w.w = w.z;
        }
        ok = mbar_wait(&bars->work_empty[work_pos.slot], work_pos.phase ^ 1u, ab, 0xB10u + work_pos.slot);
        if (!ok) break;
        bars->work[work_pos.slot] = w;
        mbar_arrive(&bars->work_full[work_pos.slot]);
        work_pos.advance(1, 2);
        if (block < 0) break;
        // its operands
        if (w.w > w.z) {
          const int tile = w.x, batch = w.y / n_own, own_head = w.y % n_own;
          const int kv_head = kPass == kWideDq ? own_head / group : own_head;
          const int4* entries = p.entries + (int64_t)batch * p.entries_per_batch;
          auto load_half_tiles = [&](uint8_t* dst, int half_bytes, const CUtensorMap* tm, uint64_t* bar, int halves, int row0,
                                     int head) {
            for (int h = 0; h < halves; ++h) tma_load_4d(dst + h * half_bytes, tm, bar, h * 64, row0, head, batch);
          };
          if (kA1Tmem) {  // two 64-row tiles through ring 1, which the compute warps carry to TMEM
            for (int sub = 0; sub < 2 && ok; ++sub) {
              ok = mbar_wait(&bars->empty1[r1.slot], r1.phase ^ 1u, ab, 0xC20u + r1.slot);
              if (!ok) break;
              mbar_arrive_expect_tx(&bars->full1[r1.slot], (uint32_t)bytes1);
              load_half_tiles(ring1 + r1.slot * bytes1, kSubHalfBytes, &tm_a1, &bars->full1[r1.slot], halves_qk,
                              tile * kTile + sub * kSub, own_head);
              r1.advance(1, n1);
            }
          }
          if (kHasDp && ok && stepped > 0) ok = mbar_wait(&bars->stat_free, (stepped - 1) & 1u, ab, 0xC30u);
          if (!ok) break;
          if (!kA1Tmem) {
            mbar_arrive_expect_tx(&bars->a1_ready, (uint32_t)(halves_qk * kHalfBytes));
            for (int sub = 0; sub < 2; ++sub)
              load_half_tiles(a1_smem + sub * kSubHalfBytes, kHalfBytes, &tm_a1, &bars->a1_ready, halves_qk,
                              tile * kTile + sub * kSub, own_head);
          }
          bool a2_due = kHasDp;  // (behind the first tile of ring 1: the first scores do not need it)
          for (int g = 0; g < heads_here && ok; ++g) {
            // streamed tiles: K / V of the kv head (dq pass) or Q / dO of q head g of the group
            const int head = kPass == kWideDq ? kv_head : kv_head * group + g;
            const int64_t stat_base = ((int64_t)batch * p.q_heads + head) * p.q_len;
            auto load_stats = [&](uint32_t slot, int row0, uint64_t* bar) {
              float* dst = stats + slot * 2 * kSub;
              bulk_load(dst, p.nlse2 + stat_base + row0, kSub * 4, bar);
              bulk_load(dst + kSub, p.delta + stat_base + row0, kSub * 4, bar);
            };
            for (int e = w.z; e < w.w && ok; ++e) {
              const int first = entries[e].x * kTile;
              for (int sub = 0; sub < 2 && ok; ++sub) {
                const int row0 = first + sub * kSub;
                ok = mbar_wait(&bars->empty1[r1.slot], r1.phase ^ 1u, ab, 0xC00u + r1.slot);
                if (!ok) break;
                constexpr bool st1 = kPass == kWideDkv || kPass == kWideDk;  // statistics ride on a held tile's barrier
                mbar_arrive_expect_tx(&bars->full1[r1.slot], (uint32_t)bytes1 + (st1 ? 2 * kSub * 4 : 0));
                load_half_tiles(ring1 + r1.slot * bytes1, kSubHalfBytes, &tm_x1, &bars->full1[r1.slot], halves_qk, row0, head);
                if (st1) load_stats(r1.slot, row0, &bars->full1[r1.slot]);
                r1.advance(1, n1);
                if (a2_due) {
                  a2_due = false;
                  mbar_arrive_expect_tx(&bars->a2_full, (uint32_t)(halves_v * kHalfBytes));
                  for (int s = 0; s < 2; ++s)
                    load_half_tiles(a2_smem + s * kSubHalfBytes, kHalfBytes, &tm_a2, &bars->a2_full, halves_v,
                                    tile * kTile + s * kSub, own_head);
                }
                ok = mbar_wait(&bars->empty2[r2.slot], r2.phase ^ 1u, ab, 0xC10u + r2.slot);
                if (!ok) break;
                constexpr bool st2 = kPass == kWideDv;
                mbar_arrive_expect_tx(&bars->full2[r2.slot], (uint32_t)bytes2 + (st2 ? 2 * kSub * 4 : 0));
                load_half_tiles(ring2 + r2.slot * bytes2, kSubHalfBytes, &tm_x2, &bars->full2[r2.slot], halves_v, row0, head);
                if (st2) load_stats(r2.slot, row0, &bars->full2[r2.slot]);
                r2.advance(1, n2);
              }
            }
          }
          ++stepped;
        }
        if (!ok) break;
        // The next tile.  Asked for when all of this one is on its way, a ring's depth ahead of the MMAs, and no earlier:
        // what a CTA has taken over, no other can take that is done before it.
        mbar_arrive_expect_tx(&bars->answer_full, 16);
        clc_request(bars->answer, &bars->answer_full);
        ok = mbar_wait(&bars->answer_full, asked & 1u, ab, 0xB20u);
        ++asked;
        if (ok) block = clc_block(bars->answer);
        fence_proxy_async_smem();  // read before the next answer overwrites it
      }
    }
  } else if (warp == kWideMmaWarp) {
    // ------------------------------------------------------------------ MMA issuer
    if (elect_one()) {
      constexpr uint32_t idesc_s = make_idesc_bf16(kTile, kSub, false, false);
      const uint32_t idesc_qk = make_idesc_bf16(kTile, halves_qk * 64, false, true);
      const uint32_t idesc_v = make_idesc_bf16(kTile, halves_v * 64, false, true);
      const uint32_t t_dp = tmem + kColDp, t_out = tmem + kColOut, t_out2 = t_out + halves_qk * 64;
      const uint32_t ring1_addr = smem_u32(ring1), ring2_addr = smem_u32(ring2);
      const SmemDesc a1 = make_smem_desc_sw128(smem_u32(a1_smem), 16, 1024), a2 = make_smem_desc_sw128(smem_u32(a2_smem), 16, 1024);
      auto t_s = [&](uint32_t n) { return tmem + (kOneS ? 0u : (n & 1u) * kSub); };
      // 128 x 64 scores: both operands K-major, K = 16 a slice, four slices a half.  (A straight run of MMAs a
      // half, the test of nk between halves: the issuing thread pays for every instruction between two MMAs.)
      auto score = [&](uint32_t d, bool a_tmem, SmemDesc da, uint32_t b0, int nk) {
        const SmemDesc db = make_smem_desc_sw128(b0, 16, 1024);
        auto slice = [&](int h, int k) {
          const SmemDesc b = desc_at(db, h * kSubHalfBytes + k * 32);
          if (a_tmem)
            umma_ts(d, tmem + kColA1 + h * 32 + k * 8, b, idesc_s, (h + k) > 0 ? 1u : 0u);
          else
            umma_ss(d, desc_at(da, h * kHalfBytes + k * 32), b, idesc_s, (h + k) > 0 ? 1u : 0u);
        };
#pragma unroll
        for (int h = 0; h < 4; ++h) {
          if (4 * h >= nk) break;
          if (4 * h + 4 <= nk) {
#pragma unroll
            for (int k = 0; k < 4; ++k) slice(h, k);
          } else {
            for (int k = 0; 4 * h + k < nk; ++k) slice(h, k);
          }
        }
      };
      // out (+)= A B: A packed in TMEM (16 columns at the start of every 32, from column a0), B a streamed tile
      // read MN-major, K = its 64 rows in four slices, N = all its columns
      auto accumulate = [&](uint32_t out, uint32_t a0, uint32_t b0, uint32_t idesc, bool acc) {
        const SmemDesc db = make_smem_desc_sw128(b0, kSubHalfBytes, 1024);
#pragma unroll
        for (int k = 0; k < 4; ++k)
          umma_ts(out, a0 + (k >> 1) * 32 + (k & 1) * 8, desc_at(db, k * 2048), idesc, (acc || k > 0) ? 1u : 0u);
      };
      bool ok = true;
      RingPos s1{0, 0};  // ring 1 where S takes its tile
      RingPos o1{0, 0};  // ring 1 where an output MMA does
      RingPos d2{0, 0};  // ring 2 where dP does
      RingPos o2{0, 0};  // ring 2 where the dv MMA does
      uint32_t ph = 0;       // parity of the sets' barriers (a tile has as many steps for one as for the other)
      uint32_t stepped = 0;  // tiles with steps so far
      for (;;) {
        int4 w;
        if (!next_work(w)) break;
        work_read();
        work_pos.advance(1, 2);
        if (w.x < 0) break;
        const uint32_t n_steps = 2u * (uint32_t)(w.w - w.z) * (uint32_t)heads_here;
        if (n_steps == 0) continue;
        ok = mbar_wait(&bars->a1_ready, stepped & 1u, ab, 0xD00u);
        if (!ok) break;
        if (kA1Tmem) {
          for (int i = 0; i < 2; ++i) {  // its two slots of ring 1 are free again
            mbar_arrive(&bars->empty1[s1.slot]);
            s1.advance(1, n1);
          }
          o1.advance(2, n1);
        }
        auto issue_s = [&](uint32_t n) {
          if (!mbar_wait(&bars->full1[s1.slot], s1.phase, ab, 0xD10u + s1.slot)) return false;
          mma_issue_fence();
          score(t_s(n), kA1Tmem, a1, ring1_addr + s1.slot * bytes1, p.nk_qk);
          tc_commit(&bars->s_full[n & 1u]);
          if (kPass == kWideDv) tc_commit(&bars->empty1[s1.slot]);
          s1.advance(1, n1);
          return true;
        };
        auto issue_dp = [&](uint32_t n) {
          if (!mbar_wait(&bars->full2[d2.slot], d2.phase, ab, 0xD20u + d2.slot)) return false;
          mma_issue_fence();
          score(t_dp, false, a2, ring2_addr + d2.slot * bytes2, p.nk_v);
          tc_commit(&bars->dp_full[n & 1u]);
          if (kPass != kWideDkv) tc_commit(&bars->empty2[d2.slot]);
          if (n + 1 == n_steps) tc_commit(&bars->stat_free);  // (the last S was issued before)
          d2.advance(1, n2);
          return true;
        };
        ok = issue_s(0);
        if (kHasDp) ok = ok && mbar_wait(&bars->a2_full, stepped & 1u, ab, 0xD01u) && issue_dp(0);
        for (uint32_t n = 0; n < n_steps && ok; ++n) {
          const uint32_t set = n & 1u;
          const bool more = n + 1 < n_steps;
          if (more) {  // the next step's scores run while this step's are worked on
            if (kOneS) ok = mbar_wait(&bars->s_free[set], ph, ab, 0xD30u);
            ok = ok && issue_s(n + 1);
            if (!ok) break;
          }
          if (n == 0 && stepped > 0) {  // the previous tile's outputs have left their columns
            ok = mbar_wait(&bars->out_free, (stepped - 1) & 1u, ab, 0xD70u);
            if (!ok) break;
          }
          if (kHasP) {
            ok = mbar_wait(&bars->p_full[set], ph, ab, 0xD40u);
            if (kPass == kWideDv) ok = ok && mbar_wait(&bars->full2[o2.slot], o2.phase, ab, 0xD50u + o2.slot);
            if (!ok) break;
            mma_issue_fence();
            accumulate(kPass == kWideDkv ? t_out2 : t_out, t_s(n), ring2_addr + o2.slot * bytes2, idesc_v, n > 0);
            tc_commit(&bars->empty2[o2.slot]);
            o2.advance(1, n2);
          }
          if (kHasDp) {
            ok = mbar_wait(&bars->ds_full[set], ph, ab, 0xD60u);
            if (!ok) break;
            mma_issue_fence();
            if (!kOneS && more) {  // dS lies over the scores: dP of the next step need not wait for the output MMA
              ok = issue_dp(n + 1);
              if (!ok) break;
            }
            accumulate(t_out, kOneS ? t_dp : t_s(n) + kDsOffset, ring1_addr + o1.slot * bytes1, idesc_qk, n > 0);
            tc_commit(&bars->empty1[o1.slot]);
            o1.advance(1, n1);
            if (kOneS && more) ok = issue_dp(n + 1);
          } else {
            o1.advance(1, n1);
          }
          ph ^= set;
        }
        if (!ok) break;
        tc_commit(&bars->acc_done);
        ++stepped;
      }
    }
  } else {
    // ------------------------------------------------------------------ compute warps
    const int cq = warp >> 2;                // 0..3: set and columns of its steps
    const int set = cq >> 1, cw = cq & 1;    // steps n % 2 = set; columns 32 cw .. 32 cw + 31 of the step
    const int wq = warp & 3;                 // TMEM lane quarter
    const int r = wq * 32 + lane;            // row within the tile: a q row (dq pass) or a kv row
    const uint32_t lane_addr = (uint32_t)(wq * 32) << 16;
    const uint32_t t_s = tmem + lane_addr + (kOneS ? 0 : set * kSub) + cw * 32;
    const uint32_t t_dp = tmem + lane_addr + kColDp + cw * 32;
    const float c = kSoftCap ? p.soft_cap * kLog2e : p.scale_log2;
    const bool has_seg = p.q_seg != nullptr;
    const uint32_t n_held = kPass == kWideDv ? n2 : n1;
    RingPos base{0, 0};    // ring of the held tile, whose barrier carries the statistics: where the current tile begins
    uint32_t ph = 0;       // parity of this set's steps
    uint32_t stepped = 0;  // tiles with steps so far

    int4 cur = make_int4(-1, 0, 0, 0);
    RingPos a1_pos{0, 0};  // ring 1: where the next tile's stationary operand comes through
    // takes the next tile, and carries its stationary operand of the scores to TMEM: row r of the tile in lane r, two
    // bf16 values a column, 64 head-dim columns a warp (every MMA that read the last tile's has completed)
    auto take_work = [&](int4& w) {
      bool ok = next_work(w);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) return false;
      if (lane == 0) work_read();
      work_pos.advance(1, 2);
      const uint32_t n_steps = w.x < 0 ? 0u : 2u * (uint32_t)(w.w - w.z) * (uint32_t)heads_here;
      if (!kA1Tmem || n_steps == 0) return true;
      RingPos pos = a1_pos;
      if (wq >= 2) pos.advance(1, n1);
      a1_pos.skip(2 + n_steps, n1);
      if (cq < halves_qk) {
        ok = mbar_wait(&bars->full1[pos.slot], pos.phase, ab, 0xE40u + pos.slot);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) return false;
        const uint8_t* src = ring1 + pos.slot * bytes1 + cq * kSubHalfBytes + (r & 63) * 128;
        uint32_t v[32];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const uint4 x = *reinterpret_cast<const uint4*>(src + ((j ^ (r & 7)) << 4));
          v[4 * j] = x.x, v[4 * j + 1] = x.y, v[4 * j + 2] = x.z, v[4 * j + 3] = x.w;
        }
        tmem_st32(tmem + lane_addr + kColA1 + cq * 32, v);
        tmem_st_wait();
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bars->a1_ready);
      return true;
    };

    bool ok = take_work(cur);
    // The dkv pass holds scores as matrix fragments, as the dkv kernel of the narrower heads does: statistics belong to columns
    // there, and a thread then needs those of 8 instead of 32.  (192, 128): causal 2 x 2048, 16 / 16
    // 256 -> 247 us a pass, 4096, 32 / 32 754 -> 751.  The dk and dv passes of wider heads lose by it: causal 8192, 16 / 8, 256
    // 2140 -> 2164.
    constexpr bool kFrag = kPass == kWideDkv;
    auto frag_at = [](int k, int hq) { return 16 * (hq >> 1) + 4 * k + 2 * (hq & 1); };  // columns 8 k, row 8 hq on
    auto load_scores = [&](uint32_t t, uint32_t (&v)[32]) {
      if constexpr (kFrag) {
        tmem_ld_frag(t, v);
        tmem_ld_frag(t + kLanes16, v + 16);
      } else {
        tmem_ld32(t, v);
      }
    };
    auto store_scores = [&](uint32_t t, const uint32_t (&pk)[16]) {
      if constexpr (kFrag) {
        tmem_st_frag(t, pk);
        tmem_st_frag(t + kLanes16, pk + 8);
      } else {
        tmem_st16(t, pk);
      }
    };
    while (ok && cur.x >= 0) {
      const int tile = cur.x, batch = cur.y / n_own, own_head = cur.y % n_own, ebeg = cur.z, eend = cur.w;
      [[maybe_unused]] const int kv_head = kPass == kWideDq ? own_head / group : own_head;
      const int4* entries = p.entries + (int64_t)batch * p.entries_per_batch;
      const uint32_t n_steps = 2u * (uint32_t)(eend - ebeg) * (uint32_t)heads_here;
      const int row = tile * kTile + (kFrag ? wq * 32 + (lane >> 2) : r);  // kFrag: the first of four, 8 apart
      int own_seg[kFrag ? 4 : 1] = {};
      RowInterval iv{INT32_MIN, INT32_MAX};
      float row_nlse2 = 0.f, row_ndelta = 0.f;
      if (kPass == kWideDq) {  // everything per row is fixed for the tile
        const int qi = p.q_sequence ? p.q_sequence[row] : row;
        iv = mask_fn_interval(p.fn, qi);
        own_seg[0] = has_seg ? p.q_seg[(int64_t)batch * p.q_len + row] : 0;
        const int64_t stat = ((int64_t)batch * p.q_heads + own_head) * p.q_len + row;
        row_nlse2 = p.nlse2[stat];
        row_ndelta = p.delta[stat];
      } else if (has_seg) {
#pragma unroll
        for (int hq = 0; hq < (kFrag ? 4 : 1); ++hq) own_seg[hq] = p.kv_seg[(int64_t)batch * p.kv_len + row + 8 * hq];
      }
      const int32_t* other_seg = has_seg ? (kPass == kWideDq ? p.kv_seg + (int64_t)batch * p.kv_len
                                                               : p.q_seg + (int64_t)batch * p.q_len)
                                         : nullptr;
      if (n_steps > 0 && kPass == kWideDk) base.skip(2, n_held);  // (its stationary operand's two slots)
      RingPos held = base;
      held.advance((uint32_t)set, n_held);
      base.skip(n_steps, n_held);

      for (int g = 0; g < heads_here && ok; ++g) {
        int4 ent_next = ebeg < eend ? entries[ebeg] : make_int4(0, 0, 0, 0);
        for (int e = ebeg; e < eend && ok; ++e) {
          const int4 ent = ent_next;
          if (e + 1 < eend) ent_next = entries[e + 1];
          const int st = ent.y & 3;
          const int c0 = ent.x * kTile + set * kSub + cw * 32;  // first column: a key (dq pass) or a query row
          // (kFrag: this thread's first two; the next are 4 words on)
          const float2* nl2 = reinterpret_cast<const float2*>(stats + held.slot * 2 * kSub + cw * 32 + (kFrag ? 2 * (lane & 3) : 0));
          const float2* dl2 = nl2 + kSub / 2;
          [[maybe_unused]] const float4* nl4 = reinterpret_cast<const float4*>(nl2);
          [[maybe_unused]] const float4* dl4 = nl4 + kSub / 4;
          ok = mbar_wait(&bars->s_full[set], ph, ab, 0xE00u);
          if (kPass != kWideDq) {
            // (behind s_full: only then has the slot's previous use, another set's perhaps, surely completed)
            ok = ok && mbar_wait(kPass == kWideDv ? &bars->full2[held.slot] : &bars->full1[held.slot], held.phase, ab, 0xE30u);
            held.advance(2, n_held);
          }
          ok = __all_sync(0xffffffffu, ok);
          if (!ok) break;
          tc_fence_after();
          float pr[32];
          {
            uint32_t v[32];
            load_scores(t_s, v);
            tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < 32; ++j) pr[j] = __uint_as_float(v[j]);
          }
          if constexpr (kOneS) {
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&bars->s_free[set]);
          }
          if constexpr (kSoftCap) {  // pr <- tanh(scale * s / cap), capped before it is masked
            tanh_all(pr, p.softcap_a);
          }
          if (st == 1) {
            if (p.fn.kind != SPLASH_MASK_TABLE) {
              if (kPass == kWideDq) {
                const int lo_rel = iv.lo <= c0 ? 0 : iv.lo - c0;
                const int hi_rel = iv.hi >= c0 + 31 ? 31 : iv.hi - c0;
#pragma unroll
                for (int j = 0; j < 32; ++j)
                  if (j < lo_rel || j > hi_rel) pr[j] = kMaskedLogit;
              } else if (!kFrag && p.q_sequence == nullptr) {
#pragma unroll
                for (int j = 0; j < 32; ++j) {
                  const RowInterval ivj = mask_fn_interval(p.fn, c0 + j);
                  if (row < ivj.lo || row > ivj.hi) pr[j] = kMaskedLogit;
                }
              } else if (!kFrag) {
#pragma unroll
                for (int j = 0; j < 32; ++j) {
                  const RowInterval ivj = mask_fn_interval(p.fn, __ldg(p.q_sequence + c0 + j));
                  if (row < ivj.lo || row > ivj.hi) pr[j] = kMaskedLogit;
                }
              } else {
#pragma unroll
                for (int k = 0; k < 4; ++k)
#pragma unroll
                  for (int u = 0; u < 2; ++u) {
                    const int q = c0 + 2 * (lane & 3) + 8 * k + u;
                    const RowInterval ivj = mask_fn_interval(p.fn, p.q_sequence == nullptr ? q : __ldg(p.q_sequence + q));
#pragma unroll
                    for (int hq = 0; hq < 4; ++hq)
                      if (row + 8 * hq < ivj.lo || row + 8 * hq > ivj.hi) pr[frag_at(k, hq) + u] = kMaskedLogit;
                  }
              }
            } else {
              // partial blocks: [id][q][kv] for the dq pass, stored transposed ([id][kv][q]) for dk / dv
              if constexpr (kFrag) {
                const int8_t* mrow = p.pmb + ((int64_t)ent.z * p.pm_bkv + (row % p.pm_bkv)) * p.pm_bq + (c0 % p.pm_bq) + 8 * (lane & 3);
                uint32_t bits = 0;  // a lane's four rows, eight columns each
#pragma unroll
                for (int hq = 0; hq < 4; ++hq) {
                  const int2 m = __ldg(reinterpret_cast<const int2*>(mrow + (int64_t)(8 * hq) * p.pm_bq));
                  bits |= (nonzero_bytes((uint32_t)m.x) | nonzero_bytes((uint32_t)m.y) << 4) << (8 * hq);
                }
#pragma unroll
                for (int k = 0; k < 4; ++k) {  // lane 4 i + k of the four that share the rows holds columns 8 k .. + 7
                  const uint32_t mine = __shfl_sync(0xffffffffu, bits, k, 4) >> (2 * (lane & 3));
#pragma unroll
                  for (int hq = 0; hq < 4; ++hq)
#pragma unroll
                    for (int u = 0; u < 2; ++u)
                      if (((mine >> (8 * hq + u)) & 1u) == 0u) pr[frag_at(k, hq) + u] = kMaskedLogit;
                }
              } else {
                const int8_t* mrow =
                    kPass == kWideDq
                        ? p.pmb + ((int64_t)ent.z * p.pm_bq + (row % p.pm_bq)) * p.pm_bkv + (c0 % p.pm_bkv)
                        : p.pmb + ((int64_t)ent.z * p.pm_bkv + (row % p.pm_bkv)) * p.pm_bq + (c0 % p.pm_bq);
                const int4* m4 = reinterpret_cast<const int4*>(mrow);
#pragma unroll
                for (int t = 0; t < 2; ++t) {
                  const int4 mv = __ldg(m4 + t);
                  const uint32_t wd[4] = {(uint32_t)mv.x, (uint32_t)mv.y, (uint32_t)mv.z, (uint32_t)mv.w};
#pragma unroll
                  for (int j = 0; j < 16; ++j)
                    if (((wd[j >> 2] >> ((j & 3) * 8)) & 0xffu) == 0u) pr[t * 16 + j] = kMaskedLogit;
                }
              }
            }
          }
          if (has_seg && !((ent.y >> 4) & 1)) {  // (bit set: the whole tile lies inside one segment)
            if constexpr (kFrag) {
#pragma unroll
              for (int k = 0; k < 4; ++k) {
                const int2 sv = __ldg(reinterpret_cast<const int2*>(other_seg + c0) + (lane & 3) + 4 * k);
#pragma unroll
                for (int hq = 0; hq < 4; ++hq) {
                  if (sv.x != own_seg[hq]) pr[frag_at(k, hq)] = kMaskedLogit;
                  if (sv.y != own_seg[hq]) pr[frag_at(k, hq) + 1] = kMaskedLogit;
                }
              }
            } else {
              const int4* sg4 = reinterpret_cast<const int4*>(other_seg + c0);
#pragma unroll
              for (int t = 0; t < 8; ++t) {
                const int4 sv = __ldg(sg4 + t);
                if (sv.x != own_seg[0]) pr[t * 4 + 0] = kMaskedLogit;
                if (sv.y != own_seg[0]) pr[t * 4 + 1] = kMaskedLogit;
                if (sv.z != own_seg[0]) pr[t * 4 + 2] = kMaskedLogit;
                if (sv.w != own_seg[0]) pr[t * 4 + 3] = kMaskedLogit;
              }
            }
          }
          // P = exp2(c * s - lse * log2 e); with a soft cap dS carries the factor 1 - tanh^2, which goes into
          // pr once P is packed (masked entries hold -1e30 in place of tanh; the clamp keeps their factor
          // finite, their p is 0)
          {
            uint32_t pk[16];
            if constexpr (kFrag) {
#pragma unroll
            for (int i = 0; i < 16; ++i) {
              const int j = frag_at(i >> 2, i & 3);
              const float2 nl = nl2[4 * (i >> 2)];
              const float2 th = make_float2(fmaxf(pr[j], -1.0f), fmaxf(pr[j + 1], -1.0f));
              const float2 x = __ffma2_rn(make_float2(pr[j], pr[j + 1]), make_float2(c, c), nl);
              pr[j] = ex2(x.x);
              pr[j + 1] = ex2(x.y);
              pk[j / 2] = pack_bf16(pr[j], pr[j + 1]);
              if constexpr (kSoftCap && kHasDp) {
                pr[j] *= fmaf(-th.x, th.x, 1.0f);
                pr[j + 1] *= fmaf(-th.y, th.y, 1.0f);
              }
            }
            } else {
#pragma unroll
              for (int t = 0; t < 8; ++t) {
                const float4 nl = kPass == kWideDq ? make_float4(row_nlse2, row_nlse2, row_nlse2, row_nlse2) : nl4[t];
                float th[4];
                if constexpr (kSoftCap && kHasDp) {
#pragma unroll
                  for (int u = 0; u < 4; ++u) th[u] = fmaxf(pr[4 * t + u], -1.0f);
                }
                const float2 xa = __ffma2_rn(make_float2(pr[4 * t + 0], pr[4 * t + 1]), make_float2(c, c), make_float2(nl.x, nl.y));
                const float2 xb = __ffma2_rn(make_float2(pr[4 * t + 2], pr[4 * t + 3]), make_float2(c, c), make_float2(nl.z, nl.w));
                pr[4 * t + 0] = ex2(xa.x);
                pr[4 * t + 1] = ex2(xa.y);
                pr[4 * t + 2] = ex2(xb.x);
                pr[4 * t + 3] = ex2(xb.y);
                pk[2 * t] = pack_bf16(pr[4 * t + 0], pr[4 * t + 1]);
                pk[2 * t + 1] = pack_bf16(pr[4 * t + 2], pr[4 * t + 3]);
                if constexpr (kSoftCap && kHasDp) {
#pragma unroll
                  for (int u = 0; u < 4; ++u) pr[4 * t + u] *= fmaf(-th[u], th[u], 1.0f);
                }
              }
            }
            if constexpr (kHasP) {
              store_scores(t_s, pk);
              tmem_st_wait();
              tc_fence_before();
              __syncwarp();
              if (lane == 0) mbar_arrive(&bars->p_full[set]);
            }
          }
          if constexpr (kHasDp) {
            ok = mbar_wait(&bars->dp_full[set], ph, ab, 0xE10u);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            tc_fence_after();
            uint32_t v[32], pk[16];
            load_scores(t_dp, v);
            tmem_ld_wait();
            if constexpr (kFrag) {
#pragma unroll
            for (int i = 0; i < 16; ++i) {
              const int j = frag_at(i >> 2, i & 3);
              const float2 nd = dl2[4 * (i >> 2)];  // -di
              const float2 ds = __fmul2_rn(make_float2(pr[j], pr[j + 1]),
                                           __fadd2_rn(make_float2(__uint_as_float(v[j]), __uint_as_float(v[j + 1])), nd));
              pk[j / 2] = pack_bf16(ds.x, ds.y);
            }
            } else {
#pragma unroll
              for (int t = 0; t < 8; ++t) {
                const float4 nd = kPass == kWideDq ? make_float4(row_ndelta, row_ndelta, row_ndelta, row_ndelta) : dl4[t];  // -di
                const float2 da = __fmul2_rn(make_float2(pr[4 * t + 0], pr[4 * t + 1]),
                                             __fadd2_rn(make_float2(__uint_as_float(v[4 * t + 0]), __uint_as_float(v[4 * t + 1])),
                                                        make_float2(nd.x, nd.y)));
                const float2 db = __fmul2_rn(make_float2(pr[4 * t + 2], pr[4 * t + 3]),
                                             __fadd2_rn(make_float2(__uint_as_float(v[4 * t + 2]), __uint_as_float(v[4 * t + 3])),
                                                        make_float2(nd.z, nd.w)));
                pk[2 * t] = pack_bf16(da.x, da.y);
                pk[2 * t + 1] = pack_bf16(db.x, db.y);
              }
            }
            store_scores(kOneS ? t_dp : t_s + kDsOffset, pk);
            tmem_st_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&bars->ds_full[set]);
          }
          ph ^= 1u;
        }
      }
      if (n_steps > 0 && ok) {
        ok = mbar_wait(&bars->acc_done, stepped & 1u, ab, 0xE20u);
        ok = __all_sync(0xffffffffu, ok);
        tc_fence_after();
        ++stepped;
      }
      if (!ok) break;
      // The next tile's scores can start before this tile's outputs are stored.
      int4 next;
      ok = take_work(next);
      if (!ok) break;
      // outputs: 32 columns at a time, the four column quarters in turn
      auto store = [&](__nv_bfloat16* out, int64_t sb, int64_t sh, int64_t ss, uint32_t t_out, int cols, float mul, bool last) {
        __nv_bfloat16* row0 = out + (int64_t)batch * sb + (int64_t)own_head * sh + (int64_t)(tile * kTile + wq * 32) * ss;
        for (int col = cq * 32; col < cols; col += 4 * 32) {
          uint32_t v[32];
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] = 0u;  // (a tile that no step touches gets zeros)
          if (n_steps > 0) {
            tmem_ld32(t_out + lane_addr + col, v);
            tmem_ld_wait();
          }
          store_rows32(row0, ss, v, mul, col, cols);
        }
        if (last && n_steps > 0) {
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&bars->out_free);
        }
      };
      store(p.out0, p.out0_sb, p.out0_sh, p.out0_ss, tmem + kColOut, kPass == kWideDv ? p.d_v : p.d_qk,
            kPass == kWideDv ? 1.0f : p.scale, kPass != kWideDkv);
      if constexpr (kPass == kWideDkv)
        store(p.out1, p.out1_sb, p.out1_sh, p.out1_ss, tmem + kColOut + halves_qk * 64, p.d_v, 1.0f, true);
      cur = next;
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == kWideMmaWarp) {
    __syncwarp();
    drain_after_give_up(&bars->abort_flag);
    tmem_dealloc(tmem, 512);
  }
}

// Slots of the two rings: two of each always fit; what is left goes to the operand that is held longer first.
static void wide_slots(int pass, int halves_qk, int halves_v, int* n1, int* n2) {
  const int a = pass == kWideDkv ? halves_qk : 0, a2 = pass == kWideDv ? 0 : halves_v;
  const int left = kWideTileBytes - (a + a2) * kHalfBytes;
  const int s1 = halves_qk * kSubHalfBytes, s2 = halves_v * kSubHalfBytes;
  *n1 = *n2 = 2;
  for (int turn = 0; turn < 2 * kWideMaxSlots; ++turn) {
    const bool first = (turn & 1) == (pass == kWideDv ? 1 : 0);
    int& n = first ? *n1 : *n2;
    if (n < kWideMaxSlots && *n1 * s1 + *n2 * s2 + (first ? s1 : s2) <= left) ++n;
  }
}

template <int kPass>
static int launch_wide_pass(const CUtensorMap& tm_a1, const CUtensorMap& tm_a2, const CUtensorMap& tm_x1,
                            const CUtensorMap& tm_x2, const BwdParams& p, bool soft_cap,
                            cudaStream_t stream) {
  if ((int64_t)p.n_rows * p.n_groups > 0x7fffffffll) return SPLASH_ERR_TOO_LARGE;
  constexpr bool kMayOneS = kPass == kWideDq || kPass == kWideDk;
  const bool one_s = kMayOneS && p.d_qk > 192;
  auto* kernel = one_s ? (soft_cap ? splash_bwd_wide_kernel<kPass, true, kMayOneS> : splash_bwd_wide_kernel<kPass, false, kMayOneS>)
                       : (soft_cap ? splash_bwd_wide_kernel<kPass, true, false> : splash_bwd_wide_kernel<kPass, false, false>);
  {
    static std::mutex attr_mu;
    static bool attr_done[64][4] = {};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return SPLASH_ERR_CUDA;
    std::lock_guard<std::mutex> lock(attr_mu);
    bool& done = attr_done[dev][(soft_cap ? 1 : 0) + (one_s ? 2 : 0)];
    if (!done) {
      if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kWideSmemBytes) != cudaSuccess)
        return SPLASH_ERR_CUDA;
      done = true;
    }
  }
  WideParams wp;
  wp.b = p;
  wide_slots(kPass, (p.d_qk + 63) / 64, (p.d_v + 63) / 64, &wp.n1, &wp.n2);
  kernel<<<(unsigned)(p.n_rows * p.n_groups), kWideThreads, kWideSmemBytes, stream>>>(tm_a1, tm_a2, tm_x1, tm_x2, wp);
  return cudaGetLastError() == cudaSuccess ? SPLASH_OK : SPLASH_ERR_CUDA;
}

int launch_bwd_wide(const CUtensorMap& tm_q, const CUtensorMap& tm_do, const CUtensorMap& tm_k,
                    const CUtensorMap& tm_v, const BwdParams& base, const SplashBwdArgs& a, bool soft_cap,
                    uint32_t launch_mask, cudaStream_t stream) {
  const int64_t B = a.q.size[0], Hq = a.q.size[1], Sq = a.q.size[2], Hkv = a.k.size[1], Skv = a.k.size[2];
  const int64_t row_bytes = 2 * (a.q.size[3] + a.v.size[3]);  // one token of k + v, or of q + do
  int st;
  BwdParams p = base;
  auto use_schedule = [&](const SplashDeviceSchedule& s) {
    p.row_ptr = s.row_ptr;
    p.entries = reinterpret_cast<const int4*>(s.entries);
    p.row_order = s.row_order;
    p.row_end = s.row_end;
    p.entries_per_batch = s.entries_per_batch;
    p.pmb = s.partial_mask_blocks;
    p.pm_bq = s.block_q > 0 ? s.block_q : kTile;
    p.pm_bkv = s.block_kv > 0 ? s.block_kv : kTile;
    p.n_rows = s.n_rows;
  };
  auto use_outputs = [&](const SplashTensor& t, const SplashTensor* u) {
    p.out0 = static_cast<__nv_bfloat16*>(t.data);
    p.out0_sb = t.stride[0];
    p.out0_sh = t.stride[1];
    p.out0_ss = t.stride[2];
    p.out1 = u ? static_cast<__nv_bfloat16*>(u->data) : nullptr;
    p.out1_sb = u ? u->stride[0] : 0;
    p.out1_sh = u ? u->stride[1] : 0;
    p.out1_ss = u ? u->stride[2] : 0;
  };
  p.dq_acc = nullptr;
  if (launch_mask & 2u) {
    use_schedule(a.sched_dq);
    use_outputs(a.dq, nullptr);
    p.n_groups = (int)(Hq * B);  // the q heads of one kv head stream the same K / V
    p.chunk_groups = chunk_groups_for(Skv * row_bytes / (Hq / Hkv), p.n_groups, Hq / Hkv);
    if ((st = launch_wide_pass<kWideDq>(tm_q, tm_do, tm_k, tm_v, p, soft_cap, stream))) return st;
  }
  if (launch_mask & 4u) {
    use_schedule(a.sched_dkv);
    p.n_groups = (int)(Hkv * B);  // the kv tiles of one (batch, kv head) stream the same Q / dO of its q heads
    p.chunk_groups = chunk_groups_for((Hq / Hkv) * Sq * row_bytes, p.n_groups, 1);
    if ((p.d_qk + 63) / 64 * 64 + (p.d_v + 63) / 64 * 64 <= kWideBothColumns) {
      use_outputs(a.dk, &a.dv);
      if ((st = launch_wide_pass<kWideDkv>(tm_k, tm_v, tm_q, tm_do, p, soft_cap, stream))) return st;
    } else {
      use_outputs(a.dk, nullptr);
      if ((st = launch_wide_pass<kWideDk>(tm_k, tm_v, tm_q, tm_do, p, soft_cap, stream))) return st;
      use_outputs(a.dv, nullptr);
      if ((st = launch_wide_pass<kWideDv>(tm_k, tm_v, tm_q, tm_do, p, soft_cap, stream))) return st;
    }
  }
  return SPLASH_OK;
}

}  // namespace sb
