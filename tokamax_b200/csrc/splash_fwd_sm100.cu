// Splash attention forward for sm_100a: bf16 (or block-scaled e4m3) Q/K/V, head_dim 128, fp32
// accumulation.
//
// One CTA owns two adjacent 128-row q tiles of one (batch, q head) and walks the kv tiles its
// schedule row lists.  Roles (384 threads):
//   warps 0-3 / 4-7 : softmax warpgroup of q tile 0 / 1 — one thread per score row
//   warp 8          : TMA producer (Q once, then a 4-slot ring of K and V tiles)
//   warp 9          : tcgen05 MMA issuer (and TMEM allocator)
//   warps 10-11     : idle; they complete the third warpgroup so registers can be handed
//                     from it to the softmax warpgroups (setmaxnreg)
// TMEM (512 columns): S0 | S1 | O0 | O1, 128 fp32 columns each.  P (bf16, two values per
// column) overwrites the first 64 columns of its S tile and feeds the PV MMA straight from TMEM.
// The two tiles ping-pong: while the softmax of tile 0 runs on the SIMT lanes, the tensor core
// computes QK^T of tile 1 and PV of the previous step.
//
// A CTA stays for several rows of the schedule: the producer takes over CTAs that have not been launched yet (cluster
// launch control), posts their rows and goes on loading; q k^T of the next row runs while the softmax warps
// store this one's outputs, 64 bytes of eight rows an instruction.  A CTA a row, each lane storing its own row, spent
// 10000 cycles between the loops of two rows.  What a row needs behind its steps is read again from shared memory, and
// the issuing thread's state is packed: kept over the step loop, they were spilled, and long rows lost what short ones
// gained.  A CTA a row -> this: window 1024, 2 x 6016, 64 / 8 heads, d 64 (10 steps a row) 469 -> 400 us; causal 4 x 8192,
// 32 / 8 heads (33 steps on average) 1.95 -> 1.84 ms; 2 x 8192 e4m3 949 -> 929 us, f16 P 973 -> 950; 32768 e4m3 with f16 P
// (129 steps) 6.82 -> 6.83 ms.  Rows that a cluster shares have a kernel of their own, splash_fwd_split_sm100.cu.
//
// Online softmax keeps a possibly stale running maximum: O and l are rescaled only when the
// new row maximum exceeds the one in use by more than 2^8, which keeps the TMEM round trip of
// O off the common path.  logsumexp is exact regardless (it is formed from the maximum in use
// and the matching l).
//
// Follows the arithmetic of the reference forward kernel
// (tokamax/_src/ops/experimental/tpu/splash_attention/splash_attention_kernel.py:299-527,
// masking :202-296) with the softmax scale applied in fp32 inside the kernel.
//
// kFp8 = true is the e4m3 prefill variant: Q, K and V hold e4m3 values with one fp32 scale per
// (batch, head, 128-token tile).  Tiles are 128 x 128 bytes (one swizzle atom wide), both MMAs run
// as kind::f8f6f4 with K = 32 per instruction, the product of the q and k tile scales is folded
// into the fp32 softmax scale of each score tile, and P is written back as e4m3 (four values per
// TMEM column) after being multiplied by 2^kFp8PShift and by the V tile's scale relative to the
// largest V scale of the (batch, kv head), so that it sits in the normal range of the format and
// never exceeds it.  There is no counterpart of this variant in the reference, which accepts
// bf16 / f32 only.
#include <mutex>

#include "splash_common.cuh"
#include "splash_fwd_steps.cuh"

namespace sb {

constexpr uint32_t kFwdWork = 4;  // a power of two

struct FwdBarriers {
  uint64_t answer[2];  // cluster launch control: what the request for the next row returned
  // rows in the order they are worked on: schedule row (-1: none left), group, first and last entry.  The softmax warps
  // keep their slot to the end of a row, the others copy it
  int4 work[kFwdWork];
  uint64_t answer_full;
  uint64_t work_full[kFwdWork], work_empty[kFwdWork];
  uint64_t q_full[2];
  uint64_t q_free;       // every q k^T of a row has completed
  uint64_t kv_full[kFwdStages];
  uint64_t kv_empty[kFwdStages];
  uint64_t s_full[2];
  uint64_t p_half[2];    // the first 64 key columns of P are in TMEM (the first half of the p v MMAs may go)
  uint64_t p_full[2];
  // a tile's O is complete: one phase a row in which the tile is live.  A phase for rows that pass the tile by would have
  // nothing to wait for: the issuing thread could complete the next one unseen
  uint64_t o_done[2];
  uint64_t vc_full[2];   // e4m3 with f16 P: a V tile has been converted to f16
  uint64_t vc_empty[2];  //                  the p v MMAs that read it have completed
  uint32_t tmem_base;
  uint32_t abort_flag;
  uint32_t early_exit;
};

// kFp8: e4m3 q / k / v with one scale per 128-token tile.  kP16 (with kFp8): the probabilities stay
// 16 bits wide — q k^T runs on the e4m3 tiles as they are, each V tile is converted once to f16 in
// shared memory (exact: e4m3 values are f16 values) by the two otherwise idle warps, and p v runs as
// an f16 MMA.  That variant meets the bf16 kernel's output bound; the all-e4m3 one does not (P
// rounded to 3 mantissa bits) but spends half the tensor time on p v.
template <bool kFp8, bool kSoftCap, bool kP16>
__global__ void __launch_bounds__(kFwdThreads, 1)
splash_fwd_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                  const __grid_constant__ CUtensorMap tm_v, const FwdParams p) {
  constexpr int kTB = kFp8 ? kFp8TileBytes : kTileBytes;  // bytes of one operand tile
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  uint8_t* q_smem = smem;                                  // 2 tiles
  static_assert(!kP16 || kFp8, "the f16-P variant is a variant of the e4m3 forward");
  uint8_t* kv_smem = smem + 2 * kTB;                       // ring
  uint8_t* vc_smem = smem + (2 + kFwdStages) * kTB;        // kP16: two f16 images of V tiles
  FwdBarriers* bars = reinterpret_cast<FwdBarriers*>(smem + fwd_operand_bytes(kFp8, kP16));

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  // schedule row, group, first and last entry of a block of the grid
  auto row_of = [&](unsigned block) {
    const CtaWork work = cta_work_at(block, p.row_order, p.n_rows, p.n_groups, p.chunk_groups, true);
    const int ebeg = p.row_ptr[work.row];
    const int eend = p.row_end ? p.row_end[(int64_t)(work.group / p.q_heads) * p.n_rows + work.row] : p.row_ptr[work.row + 1];
    return make_int4(work.row, work.group, ebeg, eend < ebeg ? ebeg : eend);
  };
  auto list_of = [&](const int4& w) { return p.entries + (int64_t)(w.y / p.q_heads) * p.entries_per_batch; };

  if (threadIdx.x == 0) {
    bars->early_exit = *reinterpret_cast<volatile uint32_t*>(p.err);
    bars->abort_flag = 0u;
    for (int i = 0; i < 2; ++i) {
      mbar_init(&bars->q_full[i], 1);
      mbar_init(&bars->s_full[i], 1);
      mbar_init(&bars->p_half[i], 4);  // one arrival per softmax warp
      mbar_init(&bars->p_full[i], 4);
      mbar_init(&bars->o_done[i], 1);
      mbar_init(&bars->vc_full[i], 2);   // one arrival per converting warp
      mbar_init(&bars->vc_empty[i], 1);
    }
    for (int s = 0; s < kFwdStages; ++s) {
      mbar_init(&bars->kv_full[s], 1);
      // K tiles sit in the even slots and are released by the MMAs that read them; V tiles sit in the
      // odd slots and, in the f16-P variant, are released by the two warps that convert them
      mbar_init(&bars->kv_empty[s], (kP16 && (s & 1)) ? 2 : 1);
    }
    for (uint32_t i = 0; i < kFwdWork; ++i) {
      mbar_init(&bars->work_full[i], 1);
      mbar_init(&bars->work_empty[i], kP16 ? 11 : 9);  // softmax warps, the issuing and the converting ones
    }
    mbar_init(&bars->answer_full, 1);
    mbar_init(&bars->q_free, 1);
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

  // The rows this CTA works on, in order: its own, then those it takes over (the producer posts both).
  uint32_t taken = 0;  // rows so far: slot and phase of the next one
  auto work_slot = [&]() { return taken % kFwdWork; };
  auto work_phase = [&]() { return (taken / kFwdWork) & 1u; };
  // Calls body(row) for each row, until it returns false: by a whole warp, or by a thread for its warp.  `hold`: the row's
  // slot is kept to the end, for body to read it again.
  auto each_row = [&](bool warp_wide, bool hold, auto body) {
    auto release = [&]() {
      if (warp_wide) __syncwarp();
      if (!warp_wide || lane == 0) mbar_arrive(&bars->work_empty[work_slot()]);
      ++taken;
    };
    for (;;) {
      bool ok = mbar_wait(&bars->work_full[work_slot()], work_phase(), ab, 0x700u + work_slot());
      if (warp_wide) ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      const int4 w = bars->work[work_slot()];
      if (w.x < 0) break;
      if (!hold) release();
      if (!body(w)) break;
      asm volatile("" : "+r"(taken));  // (the slot's addresses are worked out again, not kept over the row)
      if (hold) release();
    }
  };

  if (warp >= 8) {
   setmaxnreg_dec<kIssueRegs>();
   if (warp >= 10) {
    // Without kP16 these two warps are idle: only there to complete the third warpgroup for the
    // register hand-over.  With it they turn each e4m3 V tile (128 kv rows x 128 bytes, 16-byte
    // chunks swizzled by row & 7 as TMA wrote them) into the f16 tile the p v MMA reads MN-major:
    // two halves of 64 columns, rows of 128 bytes, the same swizzle — the layout a bf16 V tile has.
    if constexpr (kP16) {
      static_assert(kFwdStages % 2 == 0, "V tiles must keep to the odd ring slots");
      const int t = (warp - 10) * 32 + lane;
      uint32_t n = 0;
      each_row(true, false, [&](const int4& w) {
       bool ok = true;
       for (int e = w.z; e < w.w; ++e, ++n) {
        const uint32_t it = 2 * n + 1, s = it % kFwdStages, j = n & 1u;
        ok = mbar_wait(&bars->kv_full[s], (it / kFwdStages) & 1u, ab, 0x600u + s);
        if (ok) ok = mbar_wait(&bars->vc_empty[j], ((n >> 1) & 1u) ^ 1u, ab, 0x610u + j);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        const uint8_t* raw = kv_smem + s * kTB;
        uint8_t* dst = vc_smem + j * kTileBytes;
        // (four chunks at a time: causal 32768, 32 / 8 heads 6.82 -> 6.91 ms)
#pragma unroll 2
        for (int idx = t; idx < kTile * 8; idx += 64) {
          const int row = idx >> 3, c = idx & 7, x = row & 7;
          const uint4 in = *reinterpret_cast<const uint4*>(raw + row * 128 + ((c ^ x) << 4));
          uint4 lo, hi;
          e4m3x4_to_f16x4(in.x, lo.x, lo.y);
          e4m3x4_to_f16x4(in.y, lo.z, lo.w);
          e4m3x4_to_f16x4(in.z, hi.x, hi.y);
          e4m3x4_to_f16x4(in.w, hi.z, hi.w);
          uint8_t* base = dst + (c >> 2) * kHalfBytes + row * 128;
          const int c2 = (c & 3) * 2;
          *reinterpret_cast<uint4*>(base + ((c2 ^ x) << 4)) = lo;
          *reinterpret_cast<uint4*>(base + (((c2 + 1) ^ x) << 4)) = hi;
        }
        fence_proxy_async_smem();  // the MMA reads shared memory through the async proxy
        __syncwarp();
        if (lane == 0) {
          mbar_arrive(&bars->vc_full[j]);
          mbar_arrive(&bars->kv_empty[s]);
        }
       }
       return ok;
      });
    }
   } else if (warp == 8) {
    // ------------------------------------------------------------------ TMA producer
    if (elect_one()) {
      tma_prefetch_desc(&tm_q);
      tma_prefetch_desc(&tm_k);
      tma_prefetch_desc(&tm_v);
      uint32_t it = 0;
      uint32_t stepped = 0;  // rows with steps so far
      uint32_t asked = 0;
      bool ok = true;
      int block = (int)blockIdx.x;
      while (ok) {
        const int4 w = block >= 0 ? row_of((unsigned)block) : make_int4(-1, 0, 0, 0);
        ok = mbar_wait(&bars->work_empty[work_slot()], work_phase() ^ 1u, ab, 0x710u + work_slot());
        if (!ok) break;
        bars->work[work_slot()] = w;
        mbar_arrive(&bars->work_full[work_slot()]);
        ++taken;
        if (block < 0) break;
        if (w.z < w.w) {  // Q of the row, then its K and V tiles
          const int qt0 = 2 * w.x, head = w.y % p.q_heads, batch = w.y / p.q_heads;
          const int kv_head = head / (p.q_heads / p.kv_heads);
          const int4* entries = list_of(w);
          if (stepped > 0) ok = mbar_wait(&bars->q_free, (stepped - 1) & 1u, ab, 0x110u);
          if (!ok) break;
          for (int i = 0; i < 2; ++i) {
            if (qt0 + i < p.n_q_tiles) {
              uint8_t* dst = q_smem + i * kTB;
              const bool two = !kFp8 && p.d_qk > 64;  // bf16 tiles are two 64-column halves
              mbar_arrive_expect_tx(&bars->q_full[i], (kFp8 || two) ? kTB : kHalfBytes);
              tma_load_4d(dst, &tm_q, &bars->q_full[i], 0, (qt0 + i) * kTile, head, batch);
              if (two) tma_load_4d(dst + kHalfBytes, &tm_q, &bars->q_full[i], 64, (qt0 + i) * kTile, head, batch);
            }
          }
          for (int e = w.z; e < w.w && ok; ++e) {
            const int col = entries[e].x;
            for (int kv = 0; kv < 2 && ok; ++kv, ++it) {
              const uint32_t s = it % kFwdStages;
              const uint32_t ph = (it / kFwdStages) & 1u;
              ok = mbar_wait(&bars->kv_empty[s], ph ^ 1u, ab, 0x100u + s);
              if (!ok) break;
              uint8_t* dst = kv_smem + s * kTB;
              const CUtensorMap* tm = kv == 0 ? &tm_k : &tm_v;
              const bool two = !kFp8 && (kv == 0 ? p.d_qk : p.d_v) > 64;
              mbar_arrive_expect_tx(&bars->kv_full[s], (kFp8 || two) ? kTB : kHalfBytes);
              tma_load_4d(dst, tm, &bars->kv_full[s], 0, col * kTile, kv_head, batch);
              if (two) tma_load_4d(dst + kHalfBytes, tm, &bars->kv_full[s], 64, col * kTile, kv_head, batch);
            }
          }
          ++stepped;
        }
        if (!ok) break;
        // The next row.  Asked for when all of this one is on its way, two steps ahead of the MMAs, and no earlier: what a
        // CTA has taken over, no other can take that is done before it.
        mbar_arrive_expect_tx(&bars->answer_full, 16);
        clc_request(bars->answer, &bars->answer_full);
        ok = mbar_wait(&bars->answer_full, asked & 1u, ab, 0x120u);
        ++asked;
        if (ok) block = clc_block(bars->answer);
        fence_proxy_async_smem();  // read before the next answer overwrites it
      }
    }
  } else if (warp == 9) {
    // ------------------------------------------------------------------ MMA issuer
    // (e4m3 P: half as many MMAs, and the exponentials set the pace; a faster issuing thread only polls
    // more beside them: batch 2 causal 32768, 32 / 8 heads 13.02 ms behind a lane test, 13.37 ms elected)
    if (kFp8 && !kP16 ? lane == 0 : elect_one()) {
      const uint32_t idesc_pv = fwd_idesc_pv<kFp8>(p.d_v);
      const uint32_t q_addr = smem_u32(q_smem);
      const uint32_t vc_addr = smem_u32(vc_smem);
      const uint32_t kv_addr = smem_u32(kv_smem);
      auto issue_qk = [&](int i, uint32_t slot) {
        fwd_issue_qk<kFp8>(tmem + i * kTile, q_addr + i * kTB, kv_addr + slot * kTB, p.nk_qk);
        tc_commit(&bars->s_full[i]);
      };
      auto issue_pv = [&](int i, uint32_t slot, bool acc, int half) {
        fwd_issue_pv<kFp8, kP16>(tmem + 2 * kTile + i * kTile, tmem + i * kTile,
                                 kP16 ? vc_addr + slot * kTileBytes : kv_addr + slot * kTB, idesc_pv, acc, half);
      };

      // (The step loop of this thread runs in 56 registers; what it keeps is packed so that little of it is spilled.)
      uint32_t bits = 0;  // tile i: parity of its next P: bit i, of its next Q: bit 2 + i; its O is begun: bit 4 + i
      uint32_t it = 0;    // place in the ring of the step's K tile; its V tile is the next one
      each_row(false, false, [&](const int4& w) {
        int left = w.w - w.z;  // steps of the row
        if (left <= 0) return true;
        const int4* entry = list_of(w) + w.z;
        bits &= 15u;
        int nxt = entry->y;  // states of the row's two tiles in the next step
        bool ok = true;
        for (int i = 0; i < 2 && ok; ++i)
          if (2 * w.x + i < p.n_q_tiles) {
            ok = mbar_wait(&bars->q_full[i], (bits >> (2 + i)) & 1u, ab, 0x200u + i);
            bits ^= 4u << i;
          }
        if (ok) ok = mbar_wait(&bars->kv_full[it % kFwdStages], (it / kFwdStages) & 1u, ab, 0x300u);
        if (!ok) return false;
        mma_issue_fence();
        for (int i = 0; i < 2; ++i)
          if ((nxt >> (2 * i)) & 3) issue_qk(i, it % kFwdStages);
        tc_commit(&bars->kv_empty[it % kFwdStages]);
        for (bool more = true; more && ok; it += 2) {
          const int cur = nxt;
          ++entry;
          more = --left > 0;
          if (more) nxt = entry->y;
          const uint32_t vslot = (it + 1) % kFwdStages, kslot = (it + 2) % kFwdStages;
          const uint32_t vc = (it / 2) & 1u;  // kP16: which f16 image holds this step's V
          if constexpr (kP16)
            ok = mbar_wait(&bars->vc_full[vc], (it / 4) & 1u, ab, 0x340u + vc);
          else
            ok = mbar_wait(&bars->kv_full[vslot], ((it + 1) / kFwdStages) & 1u, ab, 0x310u + vslot);
          if (ok && more)
            ok = mbar_wait(&bars->kv_full[kslot], ((it + 2) / kFwdStages) & 1u, ab, 0x320u + kslot);
          if (!ok) break;
          mma_issue_fence();
          if (!more) tc_commit(&bars->q_free);
          for (int i = 0; i < 2 && ok; ++i) {
            if ((cur >> (2 * i)) & 3) {
              // (its softmax warps have read the previous row's O by then: they come to this row's P behind it)
              ok = mbar_wait(&bars->p_half[i], (bits >> i) & 1u, ab, 0x350u + i);
              if (!ok) break;
              mma_issue_fence();
              issue_pv(i, kP16 ? vc : vslot, (bits >> (4 + i)) & 1u, 0);
              ok = mbar_wait(&bars->p_full[i], (bits >> i) & 1u, ab, 0x330u + i);
              if (!ok) break;
              bits = (bits ^ (1u << i)) | (16u << i);
              mma_issue_fence();
              issue_pv(i, kP16 ? vc : vslot, true, 1);
            }
            if (i == 1) tc_commit(kP16 ? &bars->vc_empty[vc] : &bars->kv_empty[vslot]);
            if (!more && ((bits >> (4 + i)) & 1u)) tc_commit(&bars->o_done[i]);
            if (more && ((nxt >> (2 * i)) & 3)) issue_qk(i, kslot);
          }
          if (ok && more) tc_commit(&bars->kv_empty[kslot]);
        }
        return ok;
      });
    }
   }
  } else {
    // ------------------------------------------------------------------ softmax warpgroups
    setmaxnreg_inc<kSoftmaxRegs>();
    const int i = warp >> 2;           // q tile within the pair
    const int wq = warp & 3;           // TMEM lane quarter this warp may touch
    const int r = wq * 32 + lane;      // row within the tile
    const bool has_seg = p.q_seg != nullptr;
    const uint32_t lane_addr = (uint32_t)(wq * 32) << 16;
    const uint32_t t_s = tmem + lane_addr + i * kTile;
    const uint32_t t_o = tmem + lane_addr + 2 * kTile + i * kTile;
    uint32_t cnt = 0;
    uint32_t live_rows = 0;  // rows so far in which this tile was live
    each_row(true, true, [&](const int4& work) {
    const int head = work.y % p.q_heads, batch = work.y / p.q_heads, eend = work.w;
    const int kv_head = head / (p.q_heads / p.kv_heads);
    const int4* entries = list_of(work);
    const int q_tile = 2 * work.x + i;
    const bool valid = q_tile < p.n_q_tiles;
    const int q_row = valid ? q_tile * kTile + r : 0;
    const int qi = p.q_sequence ? p.q_sequence[q_row] : q_row;
    const RowInterval iv = mask_fn_interval(p.fn, qi);
    const int q_seg = has_seg ? p.q_seg[(int64_t)batch * p.q_len + q_row] : 0;
    const int32_t* kv_seg_row = has_seg ? p.kv_seg + (int64_t)batch * p.kv_len : nullptr;
    // e4m3: scores carry the q tile's and the kv tile's scale; V tiles are weighted relative to
    // the largest V scale of this (batch, kv head).
    float cq = kSoftCap ? p.soft_cap * kLog2e : p.scale_log2;  // score -> log2 units
    float v_ref = 1.f;
    const float* k_scale = nullptr;
    const float* v_scale = nullptr;
    if constexpr (kFp8) {
      const int64_t kbase = ((int64_t)batch * p.kv_heads + kv_head) * p.n_kv_tiles;
      k_scale = p.k_scale + kbase;
      v_scale = p.v_scale + kbase;
      if (valid) cq *= p.q_scale[((int64_t)batch * p.q_heads + head) * p.n_q_tiles + q_tile];
      float vm = 0.f;
      for (int t = lane; t < p.n_kv_tiles; t += 32) vm = fmaxf(vm, __ldg(v_scale + t));
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) vm = fmaxf(vm, __shfl_xor_sync(0xffffffffu, vm, off));
      v_ref = vm > 0.f ? vm : 1.f;
    }
    float m_used = -INFINITY;  // scaled (log2) units
    float m_true = kMaskedLogit;
    float l = 0.f;
    // A sink starts the row as one extra key of weight 1 at the sink logit; a fixed maximum
    // replaces the running one for the whole row (and a sink is then weighed against it).
    const bool fixed_max = !kFp8 && p.max_logit_value != nullptr;  // (refused for e4m3)
    float sink2 = -INFINITY;  // sink logit in log2 units
    if (p.sinks != nullptr) sink2 = p.sinks[head] * kLog2e;
    if (fixed_max) {
      m_used = p.max_logit_value[head] * kLog2e;
      if (p.sinks != nullptr) l = ex2(sink2 - m_used);
    } else if (p.sinks != nullptr) {
      m_used = sink2;
      l = 1.f;
    }
    bool started = false;
    bool ok = true;

    int4 ent_next = work.z < eend ? entries[work.z] : make_int4(0, 0, 0, 0);
    float ks_next = 1.f, vs_next = 1.f;
    if constexpr (kFp8) {
      if (work.z < eend) {
        ks_next = __ldg(k_scale + ent_next.x);
        vs_next = __ldg(v_scale + ent_next.x);
      }
    }
    for (int e = work.z; e < eend; ++e) {
      const int4 ent = ent_next;
      const float ks = ks_next, vs = vs_next;
      if (e + 1 < eend) {  // fetched a step ahead of its use
        ent_next = entries[e + 1];
        if constexpr (kFp8) {
          ks_next = __ldg(k_scale + ent_next.x);
          vs_next = __ldg(v_scale + ent_next.x);
        }
      }
      const float c = fmaxf(kFp8 ? cq * ks : cq, kMinScaleLog2);
      float v_share = 1.f, log_share = 0.f;
      if constexpr (kFp8) {
        v_share = fmaxf(__fdividef(vs, v_ref), 5.9604645e-8f);  // (so that a tile of zeros, scale 0, still counts in l)
        log_share = __log2f(v_share);
        asm volatile("" : "+f"(v_share), "+f"(log_share));  // (ahead of the wait for the scores)
      }
      const int st = (ent.y >> (2 * i)) & 3;
      if (st == 0) continue;
      ok = mbar_wait(&bars->s_full[i], cnt & 1u, ab, 0x400u + i);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      ++cnt;
      tc_fence_after();

      fwd_softmax_step<kFp8, kSoftCap, kP16>(p, &bars->p_half[i], &bars->p_full[i], t_s, t_o, i, lane, ent, st, c, v_share, log_share, iv,
                                             q_row, has_seg, q_seg, kv_seg_row, fixed_max, started, m_used, m_true, l);
      started = true;
    }

    // ---- epilogue: O / l -> bf16, logsumexp, max_logits
    {  // (the row's place is read again: the loop over the steps needs the registers)
    const int4 again = ld_again(&bars->work[work_slot()]);
    const int head = again.y % p.q_heads, batch = again.y / p.q_heads;
    const int q_tile = 2 * again.x + i;
    const bool valid = q_tile < p.n_q_tiles;
    const int q_row = valid ? q_tile * kTile + r : 0;
    if (ok && started) {
      ok = mbar_wait(&bars->o_done[i], live_rows++ & 1u, ab, 0x500u + i);
      ok = __all_sync(0xffffffffu, ok);
    }
    if (ok && valid) {
      tc_fence_after();
      // (context parallelism: the rows also go to the ranks that own them in the sequence-sharded layout)
      __nv_bfloat16* row0 = p.o + (int64_t)batch * p.o_sb + (int64_t)head * p.o_sh + (int64_t)(q_row - lane) * p.o_ss;
      // e4m3: O accumulated P * 2^shift * (v scale / v_ref) times the stored V values
      const bool live = l > 0.f;  // a row that met a live key, or has a sink
      const float inv = live ? (kFp8 ? v_ref * 0.015625f / l : 1.0f / l) : 0.f;
#pragma unroll
      for (int g = 0; g < 4; ++g) {
        if (g * 32 >= p.d_v) break;
        uint32_t v[32];
        if (started) {
          tmem_ld32(t_o + g * 32, v);
          tmem_ld_wait();
        } else {
#pragma unroll
          for (int j = 0; j < 32; ++j) v[j] = 0u;
        }
        if (kFp8 || p.o_peer.ptrs == nullptr)  // (no peers for e4m3)
          store_rows32(row0, p.o_ss, v, inv, g * 32, p.d_v);
        else
          store_rows32_peer(row0, p.o_ss, p.o_peer, batch, head, q_row - lane, v, inv, g * 32, p.d_v);
      }
      const float sink2 = p.sinks != nullptr ? p.sinks[head] * kLog2e : 0.f;
      store_row_stats<kFp8, kSoftCap>(p, batch, head, q_row, live, m_used, l, m_true, sink2, fixed_max);
    }
    tc_fence_before();  // O has been read, ahead of the next row's P
    }
    return ok;
    });
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

// ------------------------------------------------------------------------------------------
// host launcher
// ------------------------------------------------------------------------------------------
static FwdKernel fwd_kernel(int variant) {
  static const FwdKernel kernels[4] = {splash_fwd_kernel<false, false, false>, splash_fwd_kernel<true, false, false>,
                                       splash_fwd_kernel<false, true, false>, splash_fwd_kernel<true, false, true>};
  return kernels[variant];
}
static int fwd_smem_bytes(int variant) {
  return fwd_operand_bytes(variant & 1, variant == 3) + 1024 /*barriers*/ + 1024 /*alignment slack*/;
}

// CTAs that share a schedule row (256 query rows) of this call; the 128-wide kernels only
static int fwd_split(const SplashFwdArgs& a, const SplashShards& shards, int variant, const int32_t* clusters) {
  const int64_t q_shards = shards.q_shards > 1 ? shards.q_shards : 1;
  if (a.q_segment_ids != nullptr || (a.q_sequence != nullptr && q_shards == 1)) return 1;
  const int64_t n_rows = (a.q.size[2] / kTile * q_shards + 1) / 2;
  RowWork rw = estimate_row_work(a.mask_fn, (int)n_rows, 2 * kTile, (int)(a.k.size[2] / kTile),
                                 n_rows * a.q.size[0] * a.q.size[1] * (shards.head_shards > 1 ? shards.head_shards : 1));
  // e4m3 P: each CTA rounds its probabilities against the maximum of its own part, so that another number of CTAs moves results
  // by 1.7 % of their norm, the width of that rounding, not by the order of fp32 sums (f16 P: 0.05 %).  These rows keep to the
  // rule that they have had (1 x 4096, 8 / 8 heads: 69 us for 56).
  if (variant == 1) rw.n_rows = 0;
  return row_parts(rw, clusters, [&] {
    return cluster_capacity((const void*)fwd_split_kernel(variant), variant, kFwdThreads, fwd_split_smem_bytes(variant));
  });
}

int fwd_row_parts(const SplashFwdArgs& a, const SplashShards& shards, const int32_t* clusters) {
  for (int i = 0; i < 4; ++i)
    if (a.q.size[i] <= 0 || a.k.size[i] <= 0 || a.v.size[i] <= 0) return SPLASH_ERR_INVALID_ARGUMENT;
  if (a.q.size[2] % kTile != 0 || a.k.size[2] % kTile != 0) return SPLASH_ERR_INVALID_ARGUMENT;
  if (a.mask_fn.kind == SPLASH_MASK_CHUNKED && a.mask_fn.chunk <= 0) return SPLASH_ERR_INVALID_ARGUMENT;
  if (a.q.size[3] > kHeadDim || a.v.size[3] > kHeadDim) return 1;
  return fwd_split(a, shards, a.q.dtype == SPLASH_F8E4M3 ? 1 : (a.soft_cap != 0.f ? 2 : 0), clusters);
}

static int launch_fwd_common(const SplashFwdArgs& a, const SplashShards& shards, const float* q_scale, const float* k_scale,
                             const float* v_scale, bool fp8, bool p16, cudaStream_t stream) {
  int st;
  const bool soft_cap = a.soft_cap != 0.f;
  if (soft_cap && (fp8 || !(a.soft_cap > 0.f))) return fp8 ? SPLASH_ERR_UNSUPPORTED : SPLASH_ERR_INVALID_ARGUMENT;
  // a fixed maximum below the true one would push the narrow P formats of the e4m3 forward out of range
  if (fp8 && a.max_logit_value != nullptr) return SPLASH_ERR_UNSUPPORTED;
  if (fp8) {
    if ((st = check_e4m3_tensor(a.q)) || (st = check_e4m3_tensor(a.k)) || (st = check_e4m3_tensor(a.v)))
      return st;
    if (q_scale == nullptr || k_scale == nullptr || v_scale == nullptr) return SPLASH_ERR_INVALID_ARGUMENT;
  } else {
    if ((st = check_bf16_tensor(a.q)) || (st = check_bf16_tensor(a.k)) || (st = check_bf16_tensor(a.v)))
      return st;
  }
  if ((st = check_bf16_tensor(a.o))) return st;
  if ((st = check_peer_output(a.o_peer, a.q.size[2], a.v.size[3]))) return st;
  if (a.o_peer.ptrs != nullptr && (fp8 || a.q.size[3] > kHeadDim || a.v.size[3] > kHeadDim)) return SPLASH_ERR_UNSUPPORTED;
  const int64_t B = a.q.size[0], Hq = a.q.size[1], Sq = a.q.size[2], D = a.q.size[3];
  const int64_t Hkv = a.k.size[1], Skv = a.k.size[2];
  // Head dims: the MMA tile is 128 wide.  bf16 tensors with fewer columns (a multiple of 8, so rows
  // stay 16-byte aligned) are read in place — the TMA boxes reach past the row's end and the part
  // outside the tensor arrives as zeros, which change neither q k^T nor p v — and only the real
  // columns of the output are stored.  Head dims above 128 (up to 256) go to a forward of their
  // own (splash_fwd_wide_sm100.cu); e4m3 takes 128 only.
  const int64_t Dv = a.v.size[3];
  constexpr int64_t kMaxWideDim = 2 * kHeadDim;
  if (D > kMaxWideDim || Dv > kMaxWideDim || (fp8 && (D != kHeadDim || Dv != kHeadDim))) return SPLASH_ERR_UNSUPPORTED;
  const bool wide = D > kHeadDim || Dv > kHeadDim;
  if (D % 8 != 0 || Dv % 8 != 0 || a.k.size[3] != D) return SPLASH_ERR_INVALID_ARGUMENT;
  if (a.k.size[0] != B || a.v.size[0] != B || a.o.size[0] != B) return SPLASH_ERR_INVALID_ARGUMENT;
  if (a.v.size[1] != Hkv || a.v.size[2] != Skv || a.o.size[1] != Hq || a.o.size[2] != Sq ||
      a.o.size[3] != Dv)
    return SPLASH_ERR_INVALID_ARGUMENT;
  if (Hkv <= 0 || Hq % Hkv != 0) return SPLASH_ERR_INVALID_ARGUMENT;
  if (Sq % kTile != 0 || Skv % kTile != 0 || Sq <= 0 || Skv <= 0) return SPLASH_ERR_INVALID_ARGUMENT;
  if ((a.q_segment_ids == nullptr) != (a.kv_segment_ids == nullptr))
    return SPLASH_ERR_INVALID_ARGUMENT;
  if (a.error_record == nullptr || a.sched.row_ptr == nullptr || a.sched.entries == nullptr)
    return SPLASH_ERR_INVALID_ARGUMENT;
  const int n_q_tiles = (int)(Sq / kTile);
  if (a.sched.n_rows != (n_q_tiles + 1) / 2) return SPLASH_ERR_INVALID_ARGUMENT;
  if (a.mask_fn.kind == SPLASH_MASK_CHUNKED && a.mask_fn.chunk <= 0)
    return SPLASH_ERR_INVALID_ARGUMENT;
  if (Hq > 65535 || B > 65535 || n_q_tiles > 2 * 65535) return SPLASH_ERR_TOO_LARGE;
  if (!(a.scale > 0.f) || !(a.scale < 1.0e30f)) return SPLASH_ERR_INVALID_ARGUMENT;

  CUtensorMap tm_q, tm_k, tm_v;
  const int box_rows = wide ? kSub : kTile;
  if ((st = make_tile_tensor_map(&tm_q, a.q, box_rows)) || (st = make_tile_tensor_map(&tm_k, a.k, box_rows)) ||
      (st = make_tile_tensor_map(&tm_v, a.v, box_rows)))
    return st;

  FwdParams p;
  p.o = static_cast<__nv_bfloat16*>(a.o.data);
  p.o_sb = a.o.stride[0];
  p.o_sh = a.o.stride[1];
  p.o_ss = a.o.stride[2];
  p.o_peer = a.o_peer;
  p.d_v = (int)Dv;
  p.nk_qk = (int)((D + 15) / 16);
  p.d_qk = (int)D;
  p.lse = a.logsumexp;
  p.maxl = a.max_logits;
  p.q_seg = a.q_segment_ids;
  p.kv_seg = a.kv_segment_ids;
  p.q_sequence = a.q_sequence;
  p.row_ptr = a.sched.row_ptr;
  p.entries = reinterpret_cast<const int4*>(a.sched.entries);
  p.row_order = a.sched.row_order;
  p.row_end = a.sched.row_end;
  p.entries_per_batch = a.sched.entries_per_batch;
  p.pmb = a.sched.partial_mask_blocks;
  p.pm_bq = a.sched.block_q > 0 ? a.sched.block_q : kTile;
  p.pm_bkv = a.sched.block_kv > 0 ? a.sched.block_kv : kTile;
  p.fn = a.mask_fn;
  p.q_len = (int)Sq;
  p.kv_len = (int)Skv;
  p.q_heads = (int)Hq;
  p.kv_heads = (int)Hkv;
  p.n_q_tiles = n_q_tiles;
  p.n_rows = a.sched.n_rows;
  p.scale = a.scale;
  p.scale_log2 = a.scale * kLog2e;
  p.mask_value = a.mask_value;
  p.err = a.error_record;
  p.q_scale = q_scale;
  p.k_scale = k_scale;
  p.v_scale = v_scale;
  p.n_kv_tiles = (int)(Skv / kTile);
  p.sinks = a.sinks;
  p.max_logit_value = a.max_logit_value;
  p.soft_cap = a.soft_cap;
  p.softcap_a = soft_cap ? a.scale / a.soft_cap : 0.f;

  // The q heads of one kv head stream the same K / V (2 tensors of Skv x 128 elements).
  p.n_groups = (int)(Hq * B);
  const int64_t kv_row_bytes = fp8 ? 2 * kHeadDim : 2 * ((D > kHeadDim ? D : kHeadDim) + (Dv > kHeadDim ? Dv : kHeadDim));
  p.chunk_groups = chunk_groups_for(Skv * kv_row_bytes / (Hq / Hkv), p.n_groups, Hq / Hkv);
  if (wide) return launch_fwd_wide(tm_q, tm_k, tm_v, p, soft_cap, stream);
  if ((int64_t)p.n_rows * p.n_groups > 0x7fffffffll) return SPLASH_ERR_TOO_LARGE;
  const int variant = fp8 ? (p16 ? 3 : 1) : (soft_cap ? 2 : 0);
  p.n_split = fwd_split(a, shards, variant, nullptr);
  if (p.n_split < 0) return p.n_split;
  const bool split = p.n_split > 1;
  const FwdKernel kernel = split ? fwd_split_kernel(variant) : fwd_kernel(variant);
  const int smem = split ? fwd_split_smem_bytes(variant) : fwd_smem_bytes(variant);
  // The dynamic shared-memory attribute is per device and per kernel variant: set once, under a
  // lock (calls may come from several threads).
  if (!split) {
    static std::mutex attr_mu;
    static bool attr_done[64][4] = {};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return SPLASH_ERR_CUDA;
    std::lock_guard<std::mutex> lock(attr_mu);
    if (!attr_done[dev][variant]) {
      if (cudaFuncSetAttribute((const void*)kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess)
        return SPLASH_ERR_CUDA;
      attr_done[dev][variant] = true;
    }
  }
  const cudaError_t err = launch_clusters(kernel, (unsigned)(p.n_rows * p.n_groups), p.n_split, kFwdThreads, smem, stream,
                                          tm_q, tm_k, tm_v, p);
  return err == cudaSuccess ? SPLASH_OK : SPLASH_ERR_CUDA;
}

int launch_fwd(const SplashFwdArgs& a, const SplashShards& shards, cudaStream_t stream) {
  return launch_fwd_common(a, shards, nullptr, nullptr, nullptr, false, false, stream);
}

int launch_fwd_fp8(const SplashFwdFp8Args& a, const SplashShards& shards, cudaStream_t stream) {
  if (a.flags & ~(uint32_t)SPLASH_FP8_P_F16) return SPLASH_ERR_INVALID_ARGUMENT;
  return launch_fwd_common(a.base, shards, a.q_scale, a.k_scale, a.v_scale, true, (a.flags & SPLASH_FP8_P_F16) != 0, stream);
}

}  // namespace sb
