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
// 10000 cycles between the loops of two rows.  Window 1024, 2 x 6016, 64 / 8 heads, d 64 (10 steps a row): 478 -> 451 us;
// causal 4 x 8192, 32 / 8 heads (33 steps on average) 2.20 -> 2.12 ms; 32768 e4m3 (129 steps) no difference.
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
#include "splash_fwd_params.cuh"
#include "splash_split.cuh"

namespace sb {

struct FwdBarriers {
  uint64_t answer[2];  // cluster launch control: what the request for the next row returned
  int4 work[2];        // rows in the order they are worked on: schedule row (-1: none left), group, first and last entry
  uint64_t answer_full;
  uint64_t work_full[2], work_empty[2];
  uint64_t q_full[2];
  uint64_t q_free;       // every q k^T of a row has completed
  uint64_t kv_full[kFwdStages];
  uint64_t kv_empty[kFwdStages];
  uint64_t s_full[2];
  uint64_t p_half[2];    // the first 64 key columns of P are in TMEM (the first half of the p v MMAs may go)
  uint64_t p_full[2];
  // a tile's O is complete: one phase a row in which the tile is live (rows shared by a cluster: one phase).  A phase for
  // rows that pass the tile by would have nothing to wait for: the issuing thread could complete the next one unseen
  uint64_t o_done[2];
  uint64_t vc_full[2];   // e4m3 with f16 P: a V tile has been converted to f16
  uint64_t vc_empty[2];  //                  the p v MMAs that read it have completed
  uint32_t tmem_base;
  uint32_t abort_flag;
  uint32_t early_exit;
};

// kSplit: a CTA's part of the result lies over the operand tiles: 32 x 256 words of 16 bytes, one more row of statistics
constexpr int kPartBytes = (kHeadDim / 4 + 1) * 2 * kTile * 16;
__host__ __device__ constexpr int fwd_operand_bytes(bool fp8, bool p16, bool split) {
  const int tiles = (2 + kFwdStages) * (fp8 ? kFp8TileBytes : kTileBytes) + (p16 ? 2 * kTileBytes : 0) /*f16 V tiles*/;
  return split && tiles < kPartBytes ? kPartBytes : tiles;
}
__host__ __device__ constexpr int fwd_smem_bytes(bool fp8, bool p16, bool split) {
  return fwd_operand_bytes(fp8, p16, split) + 1024 /*barriers*/ + 1024 /*alignment slack*/;
}

__device__ __forceinline__ uint32_t pack_e4m3x4(float a, float b, float c, float d) {
  uint32_t r;
  asm("{\n\t.reg .b16 lo, hi;\n\t"
      "cvt.rn.satfinite.e4m3x2.f32 lo, %2, %1;\n\t"
      "cvt.rn.satfinite.e4m3x2.f32 hi, %4, %3;\n\t"
      "mov.b32 %0, {lo, hi};\n\t}\n"
      : "=r"(r)
      : "f"(a), "f"(b), "f"(c), "f"(d));
  return r;
}

__device__ __forceinline__ uint32_t pack_f16(float lo, float hi) {
  uint32_t r;
  asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
  return r;
}

// four e4m3 values (one 32-bit word, lowest byte first) -> four f16 values, exactly
__device__ __forceinline__ void e4m3x4_to_f16x4(uint32_t in, uint32_t& out01, uint32_t& out23) {
  asm("{\n\t.reg .b16 lo, hi;\n\t"
      "mov.b32 {lo, hi}, %2;\n\t"
      "cvt.rn.f16x2.e4m3x2 %0, lo;\n\t"
      "cvt.rn.f16x2.e4m3x2 %1, hi;\n\t}\n"
      : "=r"(out01), "=r"(out23)
      : "r"(in));
}

// logsumexp and max_logits of one row: `m` and `l` its maximum in use (log2 units) and sum, `m_true` its true maximum
template <bool kFp8, bool kSoftCap>
__device__ __forceinline__ void store_row_stats(const FwdParams& p, int batch, int head, int q_row, bool live, float m,
                                                float l, float m_true, float sink2, bool fixed_max) {
  const int64_t stat = ((int64_t)batch * p.q_heads + head) * p.q_len + q_row;
  if (p.lse) p.lse[stat] = live ? (m + log2f(l)) * kLn2 : p.mask_value;
  if (p.maxl) {
    float mv = kFp8 ? m_true * kLn2 : m_true * (kSoftCap ? p.soft_cap : p.scale);
    if (p.sinks != nullptr) mv = fmaxf(mv, sink2 * kLn2);
    if (fixed_max) mv = m * kLn2;
    p.maxl[stat] = live ? mv : p.mask_value;
  }
}

// kFp8: e4m3 q / k / v with one scale per 128-token tile.  kP16 (with kFp8): the probabilities stay
// 16 bits wide — q k^T runs on the e4m3 tiles as they are, each V tile is converted once to f16 in
// shared memory (exact: e4m3 values are f16 values) by the two otherwise idle warps, and p v runs as
// an f16 MMA.  That variant meets the bf16 kernel's output bound; the all-e4m3 one does not (P
// rounded to 3 mantissa bits) but spends half the tensor time on p v.
//
// kSplit: a cluster of 2 .. 8 CTAs shares one schedule row, each taking its part of the row's kv tiles
// as if the row held nothing else.  Afterwards every CTA leaves its O (fp32), maximum and sum in its
// own shared memory (the ring is free by then), and the cluster adds them up over distributed shared
// memory, each CTA a share of the columns: no scratch in global memory, no second launch, and the
// order of the additions is fixed.  For grids that leave SMs idle; split_for() holds the rule.
template <bool kFp8, bool kSoftCap, bool kP16, bool kSplit>
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
  FwdBarriers* bars = reinterpret_cast<FwdBarriers*>(smem + fwd_operand_bytes(kFp8, kP16, kSplit));

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const unsigned rank = kSplit ? cluster_rank() : 0u;
  // schedule row, group, first and last entry of a block of the grid
  auto row_of = [&](unsigned block) {
    const CtaWork work = cta_work_at(block, p.row_order, p.n_rows, p.n_groups, p.chunk_groups, true);
    const int ebeg = p.row_ptr[work.row];
    const int eend = p.row_end ? p.row_end[(int64_t)(work.group / p.q_heads) * p.n_rows + work.row] : p.row_ptr[work.row + 1];
    return make_int4(work.row, work.group, ebeg, eend < ebeg ? ebeg : eend);
  };
  auto list_of = [&](const int4& w) { return p.entries + (int64_t)(w.y / p.q_heads) * p.entries_per_batch; };
  // the entries of this CTA in a row, and the first of them (a cluster's row: looked up here, under the set-up of
  // barriers and TMEM)
  int4 own = make_int4(0, 0, 0, 0);
  if constexpr (kSplit) own = row_of(blockIdx.x / p.n_split);
  const PartWalk<kSplit> own_walk(list_of(own), own.z, own.w, p.n_split);
  int own_first = 0;
  if constexpr (kSplit) own_first = own_walk.first(own_walk.offset((int)rank));
  auto walk_of = [&](const int4& w) {
    if constexpr (kSplit) return own_walk;
    return PartWalk<kSplit>(list_of(w), w.z, w.w, p.n_split);
  };
  auto first_of = [&](const int4& w) { return kSplit ? own_first : w.z; };

  if (threadIdx.x == 0) {
    bars->early_exit = *reinterpret_cast<volatile uint32_t*>(p.err);
    bars->abort_flag = kSplit ? bars->early_exit : 0u;  // (read by the other CTAs of the cluster)
    for (int i = 0; i < 2; ++i) {
      mbar_init(&bars->q_full[i], 1);
      mbar_init(&bars->s_full[i], 1);
      mbar_init(&bars->p_half[i], 4);  // one arrival per softmax warp
      mbar_init(&bars->p_full[i], 4);
      mbar_init(&bars->o_done[i], 1);
      mbar_init(&bars->work_full[i], 1);
      mbar_init(&bars->work_empty[i], kP16 ? 11 : 9);  // softmax warps, the issuing and the converting ones
      mbar_init(&bars->vc_full[i], 2);   // one arrival per converting warp
      mbar_init(&bars->vc_empty[i], 1);
    }
    for (int s = 0; s < kFwdStages; ++s) {
      mbar_init(&bars->kv_full[s], 1);
      // K tiles sit in the even slots and are released by the MMAs that read them; V tiles sit in the
      // odd slots and, in the f16-P variant, are released by the two warps that convert them
      mbar_init(&bars->kv_empty[s], (kP16 && (s & 1)) ? 2 : 1);
    }
    mbar_init(&bars->answer_full, 1);
    mbar_init(&bars->q_free, 1);
    mbar_fence_init();
  }
  __syncthreads();
  if (bars->early_exit != 0) {  // an earlier CTA already reported a fault
    if constexpr (kSplit) {  // the others may not have seen it: no CTA leaves while its shared memory may be read
      cluster_sync();
      cluster_sync();
    }
    return;
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

  // The rows this CTA works on, in order: its own, then those it takes over (the producer posts both).  A CTA of a
  // cluster has the cluster's row and no other.
  RingPos work_pos{0, 0};
  auto next_work = [&](int4& w, bool warp_wide) {  // by a whole warp, or by a thread for its warp
    if constexpr (kSplit) {  // (whose loops end behind it)
      w = own;
      return true;
    }
    bool ok = mbar_wait(&bars->work_full[work_pos.slot], work_pos.phase, ab, 0x700u + work_pos.slot);
    if (warp_wide) ok = __all_sync(0xffffffffu, ok);
    if (!ok) return false;
    w = bars->work[work_pos.slot];
    if (warp_wide) __syncwarp();
    if (!warp_wide || lane == 0) mbar_arrive(&bars->work_empty[work_pos.slot]);
    work_pos.advance(1, 2);
    return w.x >= 0;
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
      bool ok = true;
      int4 w;
      while (ok && next_work(w, true)) {
       const int eend = w.w;
       const PartWalk<kSplit> walk = walk_of(w);
       for (int e = first_of(w); e < eend; e = walk.next(e), ++n) {
        const uint32_t it = 2 * n + 1, s = it % kFwdStages, j = n & 1u;
        ok = mbar_wait(&bars->kv_full[s], (it / kFwdStages) & 1u, ab, 0x600u + s);
        if (ok) ok = mbar_wait(&bars->vc_empty[j], ((n >> 1) & 1u) ^ 1u, ab, 0x610u + j);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        const uint8_t* raw = kv_smem + s * kTB;
        uint8_t* dst = vc_smem + j * kTileBytes;
#pragma unroll 4
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
       if (kSplit) break;
      }
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
      for (;;) {
        int4 w = own;
        if constexpr (!kSplit) {
          w = block >= 0 ? row_of((unsigned)block) : make_int4(-1, 0, 0, 0);
          ok = mbar_wait(&bars->work_empty[work_pos.slot], work_pos.phase ^ 1u, ab, 0x710u + work_pos.slot);
          if (!ok) break;
          bars->work[work_pos.slot] = w;
          mbar_arrive(&bars->work_full[work_pos.slot]);
          work_pos.advance(1, 2);
          if (block < 0) break;
        }
        const int qt0 = 2 * w.x, head = w.y % p.q_heads, batch = w.y / p.q_heads, eend = w.w;
        const int kv_head = head / (p.q_heads / p.kv_heads);
        const int4* entries = list_of(w);
        const PartWalk<kSplit> walk = walk_of(w);
        const int efirst = first_of(w);
        if (efirst < eend) {
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
          ++stepped;
        }
        for (int e = efirst; e < eend && ok; e = walk.next(e)) {
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
        if (!ok || kSplit) break;
        // The next row.  Asked for when all of this one is on its way, two steps ahead of the MMAs, and no earlier: what a
        // CTA has taken over, no other can take that is done before it.
        mbar_arrive_expect_tx(&bars->answer_full, 16);
        clc_request(bars->answer, &bars->answer_full);
        ok = mbar_wait(&bars->answer_full, asked & 1u, ab, 0x120u);
        if (!ok) break;
        ++asked;
        block = clc_block(bars->answer);
        fence_proxy_async_smem();  // read before the next answer overwrites it
      }
    }
  } else if (warp == 9) {
    // ------------------------------------------------------------------ MMA issuer
    // (e4m3 P: half as many MMAs, and the exponentials set the pace; a faster issuing thread only polls
    // more beside them: batch 2 causal 32768, 32 / 8 heads 13.02 ms behind a lane test, 13.37 ms elected)
    if (kFp8 && !kP16 ? lane == 0 : elect_one()) {
      constexpr uint32_t idesc_qk =
          kFp8 ? make_idesc_e4m3(kTile, kTile, false, false) : make_idesc_bf16(kTile, kTile, false, false);
      // N of p v: the output's columns — 128, or 64 when v has at most 64 (half the MMA work; the
      // V tile's second half is then neither loaded nor read)
      const int n_pv = (!kFp8 && p.d_v <= 64) ? 64 : kHeadDim;
      // (kind::f16 with format code 0 for A and B is f16 x f16: the same bits as the e4m3 descriptor)
      const uint32_t idesc_pv = kFp8 ? make_idesc_e4m3(kTile, kHeadDim, false, true)
                                     : make_idesc_bf16(kTile, n_pv, false, true);
      const uint32_t q_addr = smem_u32(q_smem);
      const uint32_t vc_addr = smem_u32(vc_smem);
      const uint32_t kv_addr = smem_u32(kv_smem);
      // S_i = Q_i K^T : both operands K-major.  bf16: eight K=16 slices across two swizzle
      // halves; e4m3: four K=32 slices inside the single 128-byte-wide tile.
      auto issue_qk = [&](int i, uint32_t slot) {
        const uint32_t a0 = q_addr + i * kTB;
        const uint32_t b0 = kv_addr + slot * kTB;
        const SmemDesc da = make_smem_desc_sw128(a0, 16, 1024), db = make_smem_desc_sw128(b0, 16, 1024);
        if constexpr (kFp8) {
#pragma unroll
          for (int k = 0; k < 4; ++k)
            umma_ss_f8(tmem + i * kTile, desc_at(da, k * 32), desc_at(db, k * 32), idesc_qk, k > 0 ? 1u : 0u);
        } else {
#pragma unroll
          for (int k = 0; k < 8; ++k) {
            // head dims below 128: the remaining slices multiply zeros (nk_qk == 8 is tested first so
            // that the full-width path stays a straight run of eight MMAs)
            if (p.nk_qk != 8 && k >= p.nk_qk) break;
            const uint32_t off = (k >> 2) * kHalfBytes + (k & 3) * 32;
            umma_ss(tmem + i * kTile, desc_at(da, off), desc_at(db, off), idesc_qk, k > 0 ? 1u : 0u);
          }
        }
        tc_commit(&bars->s_full[i]);
      };
      // O_i (+)= P_i V : A from TMEM, B = V tile read MN-major (head_dim contiguous):
      // 8 kv rows x 128 B per core group (SBO 1024).  bf16: 64-column halves 16 KiB apart (LBO),
      // K=16 slices 2 KiB apart; e4m3: the 128 columns fit one 128-byte row, K=32 slices 4 KiB
      // apart, P packed four values per TMEM column.
      // `half` 0 / 1: the K slices over the first / last 64 key columns of P (the softmax warps hand
      // P over in two halves, so that the first MMAs run while the second half is still being made)
      auto issue_pv = [&](int i, uint32_t slot, bool acc, int half) {
        const uint32_t b0 = kP16 ? vc_addr + slot * kTileBytes : kv_addr + slot * kTB;
        if constexpr (kFp8 && !kP16) {
          const SmemDesc db = make_smem_desc_sw128(b0, 16, 1024);
#pragma unroll
          for (int kk = 0; kk < 2; ++kk) {
            const int k = half * 2 + kk;
            umma_ts_f8(tmem + 2 * kTile + i * kTile, tmem + i * kTile + k * 8, desc_at(db, k * 4096), idesc_pv,
                       (acc || k > 0) ? 1u : 0u);
          }
        } else {
          const SmemDesc db = make_smem_desc_sw128(b0, kHalfBytes, 1024);
#pragma unroll
          for (int kk = 0; kk < 4; ++kk) {
            const int k = half * 4 + kk;
            umma_ts(tmem + 2 * kTile + i * kTile, tmem + i * kTile + k * 8, desc_at(db, k * 2048), idesc_pv,
                    (acc || k > 0) ? 1u : 0u);
          }
        }
      };

      uint32_t pcnt[2] = {0, 0};
      uint32_t qcnt[2] = {0, 0};   // Q tiles so far
      uint32_t it0 = 0;            // ring slots of the rows before this one
      bool ok = true;
      int4 w;
      while (ok && next_work(w, false)) {
        const int4* entries = list_of(w);
        const int ebeg = w.z, eend = w.w;
        const PartWalk<kSplit> walk = walk_of(w);
        const int efirst = first_of(w);
        if (efirst >= eend) {
          if (kSplit) break;
          continue;
        }
        const int n_ent = eend - ebeg;
        int e = efirst;
        bool started[2] = {false, false};
        const int4 e0 = entries[efirst];
        for (int i = 0; i < 2 && ok; ++i)
          if (2 * w.x + i < p.n_q_tiles) ok = mbar_wait(&bars->q_full[i], qcnt[i]++ & 1u, ab, 0x200u + i);
        if (ok) ok = mbar_wait(&bars->kv_full[it0 % kFwdStages], (it0 / kFwdStages) & 1u, ab, 0x300u);
        if (!ok) break;
        mma_issue_fence();
        for (int i = 0; i < 2; ++i)
          if ((e0.y >> (2 * i)) & 3) issue_qk(i, it0 % kFwdStages);
        tc_commit(&bars->kv_empty[it0 % kFwdStages]);
        int4 nxt = e0;
        uint32_t n = 0;
        for (bool more = true; more && ok; ++n) {
          const int4 cur = nxt;
          if constexpr (kSplit) e = walk.next(e);
          const bool has_next = kSplit ? e < eend : (int)n + 1 < n_ent;
          more = has_next;
          if (has_next) nxt = entries[kSplit ? e : ebeg + (int)n + 1];
          const uint32_t itv = it0 + 2 * n + 1, itk = it0 + 2 * n + 2;
          const uint32_t vslot = itv % kFwdStages, kslot = itk % kFwdStages;
          const uint32_t step = it0 / 2 + n, vc = step & 1u;  // kP16: which f16 image holds this step's V
          if constexpr (kP16)
            ok = mbar_wait(&bars->vc_full[vc], (step >> 1) & 1u, ab, 0x340u + vc);
          else
            ok = mbar_wait(&bars->kv_full[vslot], (itv / kFwdStages) & 1u, ab, 0x310u + vslot);
          if (ok && has_next)
            ok = mbar_wait(&bars->kv_full[kslot], (itk / kFwdStages) & 1u, ab, 0x320u + kslot);
          if (!ok) break;
          mma_issue_fence();
          if (!kSplit && !has_next) tc_commit(&bars->q_free);
          for (int i = 0; i < 2 && ok; ++i) {
            if ((cur.y >> (2 * i)) & 3) {
              // (its softmax warps have read the previous row's O by then: they come to this row's P behind it)
              ok = mbar_wait(&bars->p_half[i], pcnt[i] & 1u, ab, 0x350u + i);
              if (!ok) break;
              mma_issue_fence();
              issue_pv(i, kP16 ? vc : vslot, started[i], 0);
              ok = mbar_wait(&bars->p_full[i], pcnt[i] & 1u, ab, 0x330u + i);
              if (!ok) break;
              ++pcnt[i];
              mma_issue_fence();
              issue_pv(i, kP16 ? vc : vslot, true, 1);
              started[i] = true;
            }
            if (i == 1) tc_commit(kP16 ? &bars->vc_empty[vc] : &bars->kv_empty[vslot]);
            if (!kSplit && !has_next && started[i]) tc_commit(&bars->o_done[i]);
            if (has_next && ((nxt.y >> (2 * i)) & 3)) issue_qk(i, kslot);
          }
          if (ok && has_next) tc_commit(&bars->kv_empty[kslot]);
        }
        if constexpr (kSplit) {  // the parts go over the operand tiles: not before both tiles' MMAs have read them
          tc_commit(&bars->o_done[0]);
          tc_commit(&bars->o_done[1]);
        }
        it0 += 2 * n;
        if (kSplit) break;
      }
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
    bool ok = true;
    int4 work;
    while (ok && next_work(work, true)) {
    const int head = work.y % p.q_heads, batch = work.y / p.q_heads, eend = work.w;
    const int kv_head = head / (p.q_heads / p.kv_heads);
    const int4* entries = list_of(work);
    const PartWalk<kSplit> walk = walk_of(work);
    const int efirst = first_of(work);
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
    // e4m3 P must stay below 448; f16 P (times 2^6) below 65504; bf16 P has the range of fp32
    constexpr float kThreshold = (kFp8 && !kP16) ? kFp8RescaleThreshold : kRescaleThreshold;

    float m_used = -INFINITY;  // scaled (log2) units
    float m_true = kMaskedLogit;
    float l = 0.f;
    // A sink starts the row as one extra key of weight 1 at the sink logit; a fixed maximum
    // replaces the running one for the whole row (and a sink is then weighed against it).
    const bool fixed_max = p.max_logit_value != nullptr;
    float sink2 = -INFINITY;  // sink logit in log2 units
    if (p.sinks != nullptr) sink2 = p.sinks[head] * kLog2e;
    const bool own_sink = p.sinks != nullptr && rank == 0;  // one CTA of a cluster counts it
    if (fixed_max) {
      m_used = p.max_logit_value[head] * kLog2e;
      if (own_sink) l = ex2(sink2 - m_used);
    } else if (own_sink) {
      m_used = sink2;
      l = 1.f;
    }
    bool started = false;

    int4 ent_next = efirst < eend ? entries[efirst] : make_int4(0, 0, 0, 0);
    float ks_next = 1.f, vs_next = 1.f;
    if constexpr (kFp8) {
      if (efirst < eend) {
        ks_next = __ldg(k_scale + ent_next.x);
        vs_next = __ldg(v_scale + ent_next.x);
      }
    }
    int e_last = 0, x_due = ent_next.x, e_probe = efirst;
    for (int e = efirst; e < eend; e = kSplit ? e_probe : e + 1) {
      if constexpr (kSplit) {
        if (ent_next.x != x_due) {  // a gap in the row
          e = walk.find(e_last + 1, x_due);
          if (e >= eend) break;
          ent_next = entries[e];
          if constexpr (kFp8) {
            ks_next = __ldg(k_scale + ent_next.x);
            vs_next = __ldg(v_scale + ent_next.x);
          }
        }
        e_last = e;
        x_due = ent_next.x + walk.n;
        e_probe = walk.probe(e, x_due);
      }
      const int e_next = kSplit ? e_probe : e + 1;
      const int4 ent = ent_next;
      const float ks = ks_next, vs = vs_next;
      if (e_next < eend) {  // fetched a step ahead of its use
        ent_next = entries[e_next];
        if constexpr (kFp8) {
          ks_next = __ldg(k_scale + ent_next.x);
          vs_next = __ldg(v_scale + ent_next.x);
        }
      }
      const float c = fmaxf(kFp8 ? cq * ks : cq, kMinScaleLog2);
      const int st = (ent.y >> (2 * i)) & 3;
      if (st == 0) continue;
      ok = mbar_wait(&bars->s_full[i], cnt & 1u, ab, 0x400u + i);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      ++cnt;
      tc_fence_after();

      float s[kTile];
      {
        uint32_t v0[32], v1[32], v2[32], v3[32];
        tmem_ld32(t_s, v0);
        tmem_ld32(t_s + 32, v1);
        tmem_ld32(t_s + 64, v2);
        tmem_ld32(t_s + 96, v3);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 32; ++j) {
          s[j] = __uint_as_float(v0[j]);
          s[32 + j] = __uint_as_float(v1[j]);
          s[64 + j] = __uint_as_float(v2[j]);
          s[96 + j] = __uint_as_float(v3[j]);
        }
      }
      if constexpr (kSoftCap) {
        // s <- tanh(scale * s / cap) before masking (reference :202-296 caps, then masks); the
        // factor cap * log2(e) that follows is `c`.
#pragma unroll
        for (int j = 0; j < kTile; ++j) s[j] = tanh_ex2(s[j] * p.softcap_a);
      }
      const int kv0 = ent.x * kTile;
      if (st == 1) {
        if (p.fn.kind != SPLASH_MASK_TABLE) {
          const int lo_rel = iv.lo <= kv0 ? 0 : iv.lo - kv0;
          const int hi_rel = iv.hi >= kv0 + (kTile - 1) ? kTile - 1 : iv.hi - kv0;
#pragma unroll
          for (int j = 0; j < kTile; ++j)
            if (j < lo_rel || j > hi_rel) s[j] = kMaskedLogit;
        } else {
          const int pid = i == 0 ? ent.z : ent.w;
          const int8_t* mrow = p.pmb + ((int64_t)pid * p.pm_bq + (q_row % p.pm_bq)) * p.pm_bkv +
                               (kv0 % p.pm_bkv);
          const int4* m4 = reinterpret_cast<const int4*>(mrow);
#pragma unroll
          for (int g = 0; g < 8; ++g) {
            const int4 mv = __ldg(m4 + g);
            const uint32_t w[4] = {(uint32_t)mv.x, (uint32_t)mv.y, (uint32_t)mv.z, (uint32_t)mv.w};
#pragma unroll
            for (int j = 0; j < 16; ++j)
              if (((w[j >> 2] >> ((j & 3) * 8)) & 0xffu) == 0u) s[g * 16 + j] = kMaskedLogit;
          }
        }
      }
      if (has_seg && !((ent.y >> (4 + i)) & 1)) {  // (bit set: the whole tile lies inside one segment)
        const int4* sg4 = reinterpret_cast<const int4*>(kv_seg_row + kv0);
#pragma unroll
        for (int g = 0; g < 32; ++g) {
          const int4 sv = __ldg(sg4 + g);
          if (sv.x != q_seg) s[g * 4 + 0] = kMaskedLogit;
          if (sv.y != q_seg) s[g * 4 + 1] = kMaskedLogit;
          if (sv.z != q_seg) s[g * 4 + 2] = kMaskedLogit;
          if (sv.w != q_seg) s[g * 4 + 3] = kMaskedLogit;
        }
      }

      // The softmax warps are bound by instruction issue, so the per-element work uses the
      // two-wide fp32 instructions of sm_100 (fma / add on register pairs) and three-input max.
      float mx0 = max3(s[0], s[1], s[2]), mx1 = max3(s[3], s[4], s[5]);
      float mx2 = max3(s[6], s[7], s[8]), mx3 = max3(s[9], s[10], s[11]);
#pragma unroll
      for (int j = 12; j < kTile - 4; j += 8) {
        mx0 = max3(mx0, s[j], s[j + 1]);
        mx1 = max3(mx1, s[j + 2], s[j + 3]);
        mx2 = max3(mx2, s[j + 4], s[j + 5]);
        mx3 = max3(mx3, s[j + 6], s[j + 7]);
      }
      mx0 = max3(mx0, s[kTile - 4], s[kTile - 3]);
      mx1 = max3(mx1, s[kTile - 2], s[kTile - 1]);
      const float mx = fmaxf(fmaxf(mx0, mx1), fmaxf(mx2, mx3));
      const float m_new = fmaxf(mx * c, kLogitFloor);
      m_true = fmaxf(m_true, kFp8 ? m_new : mx);  // e4m3: log2 units (the scale varies by tile)
      const bool need = !fixed_max && m_new > m_used + kThreshold;
      if (__any_sync(0xffffffffu, need)) {
        const float m_next = fmaxf(m_used, m_new);
        const float alpha = ex2(m_used - m_next);
        l *= alpha;
        if (started) {
          uint32_t v[32];
#pragma unroll
          for (int g = 0; g < 4; ++g) {
            tmem_ld32(t_o + g * 32, v);
            tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < 32; ++j) v[j] = __float_as_uint(__uint_as_float(v[j]) * alpha);
            tmem_st32(t_o + g * 32, v);
          }
        }
        m_used = m_next;
      }

      float ls0 = 0.f, ls1 = 0.f;
      if constexpr (kP16) {
        // as the e4m3 branch below, but P stays 16 bits wide (f16: 11 significant bits; the factor
        // 2^6 keeps the small weights out of the subnormals, 2^(6+8) is the largest value written)
        const float r = fmaxf(__fdividef(vs, v_ref), 5.9604645e-8f);
        const float m_sub = m_used - kFp8PShift - __log2f(r);
#pragma unroll
        for (int g = 0; g < 4; ++g) {
          uint32_t pk[16];
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            const float p0 = ex2(fmaf(s[g * 32 + 2 * j], c, -m_sub));
            const float p1 = ex2(fmaf(s[g * 32 + 2 * j + 1], c, -m_sub));
            ls0 += p0;
            ls1 += p1;
            pk[j] = pack_f16(p0, p1);
          }
          tmem_st16(t_s + g * 16, pk);
          if (g == 1) {  // the first 64 key columns are in place
            tmem_st_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&bars->p_half[i]);
          }
        }
        l += (ls0 + ls1) * __fdividef(0.015625f, r);
      } else if constexpr (kFp8) {
        // P * 2^shift * r with r = v scale / largest v scale in (0, 1]; r is floored so that a
        // tile of zeros (scale 0) still counts in l.
        const float r = fmaxf(__fdividef(vs, v_ref), 5.9604645e-8f);
        const float m_sub = m_used - kFp8PShift - __log2f(r);
#pragma unroll
        for (int g = 0; g < 2; ++g) {
          uint32_t pk[16];
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            const float p0 = ex2(fmaf(s[g * 64 + 4 * j], c, -m_sub));
            const float p1 = ex2(fmaf(s[g * 64 + 4 * j + 1], c, -m_sub));
            const float p2 = ex2(fmaf(s[g * 64 + 4 * j + 2], c, -m_sub));
            const float p3 = ex2(fmaf(s[g * 64 + 4 * j + 3], c, -m_sub));
            ls0 += p0 + p2;
            ls1 += p1 + p3;
            pk[j] = pack_e4m3x4(p0, p1, p2, p3);
          }
          tmem_st16(t_s + g * 16, pk);
          if (g == 0) {  // the first 64 key columns are in place
            tmem_st_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&bars->p_half[i]);
          }
        }
        l += (ls0 + ls1) * __fdividef(0.015625f, r);  // back to exp2(s - m) units (2^-6 / r)
      } else {
        const float2 c2 = make_float2(c, c), nm2 = make_float2(-m_used, -m_used);
        float2 lsa = make_float2(0.f, 0.f), lsb = make_float2(0.f, 0.f);
#pragma unroll
        for (int g = 0; g < 4; ++g) {
          uint32_t pk[16];
#pragma unroll
          for (int j = 0; j < 16; j += 2) {
            const float2 xa = __ffma2_rn(make_float2(s[g * 32 + 2 * j], s[g * 32 + 2 * j + 1]), c2, nm2);
            const float2 xb = __ffma2_rn(make_float2(s[g * 32 + 2 * j + 2], s[g * 32 + 2 * j + 3]), c2, nm2);
            const float2 pa = make_float2(ex2(xa.x), ex2(xa.y));
            const float2 pb = make_float2(ex2(xb.x), ex2(xb.y));
            lsa = __fadd2_rn(lsa, pa);
            lsb = __fadd2_rn(lsb, pb);
            pk[j] = pack_bf16(pa.x, pa.y);
            pk[j + 1] = pack_bf16(pb.x, pb.y);
          }
          tmem_st16(t_s + g * 16, pk);
          if (g == 1) {  // the first 64 key columns are in place
            tmem_st_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&bars->p_half[i]);
          }
        }
        ls0 = lsa.x + lsb.x;
        ls1 = lsa.y + lsb.y;
        l += ls0 + ls1;
      }
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bars->p_full[i]);
      started = true;
    }

    // ---- epilogue: O / l -> bf16, logsumexp, max_logits
    if (ok && (kSplit ? efirst < eend : started)) {
      ok = mbar_wait(&bars->o_done[i], live_rows++ & 1u, ab, 0x500u + i);
      ok = __all_sync(0xffffffffu, ok);
    }
    if constexpr (kSplit) {
      // this CTA's part of the row, [column / 4][row of the pair] in 16-byte words, then its statistics
      if (ok && valid) {
        tc_fence_after();
        float4* part = reinterpret_cast<float4*>(smem) + threadIdx.x;
#pragma unroll
        for (int g = 0; g < 4; ++g) {
          uint32_t v[32];
          if (started) {
            tmem_ld32(t_o + g * 32, v);
            tmem_ld_wait();
          } else {
#pragma unroll
            for (int j = 0; j < 32; ++j) v[j] = 0u;
          }
#pragma unroll
          for (int j = 0; j < 8; ++j)
            part[(g * 8 + j) * 2 * kTile] = make_float4(__uint_as_float(v[4 * j]), __uint_as_float(v[4 * j + 1]),
                                                        __uint_as_float(v[4 * j + 2]), __uint_as_float(v[4 * j + 3]));
        }
        part[kHeadDim / 4 * 2 * kTile] = make_float4(m_used, l, m_true, 0.f);
      }
      tc_fence_before();
      cluster_sync();  // (with the same call of the third warpgroup below)
      bool good = valid;
      float weight[kMaxSplit];
      float top = -INFINITY, sum = 0.f, m_all = kMaskedLogit;
#pragma unroll
      for (int s = 0; s < kMaxSplit; ++s) {
        weight[s] = 0.f;
        if (s < p.n_split) good = good && cluster_ld_u32(cluster_addr(&bars->abort_flag, s)) == 0u;
      }
      if (good) {
        const float4* part = reinterpret_cast<const float4*>(smem) + threadIdx.x;
        float4 st[kMaxSplit];
#pragma unroll
        for (int s = 0; s < kMaxSplit; ++s) {
          st[s] = make_float4(-INFINITY, 0.f, kMaskedLogit, 0.f);
          if (s < p.n_split) st[s] = cluster_ld_v4(cluster_addr(part + kHeadDim / 4 * 2 * kTile, s));
          top = fmaxf(top, st[s].x);  // (-inf: nothing seen; the floor: dead keys only, as in a row left whole)
          m_all = fmaxf(m_all, st[s].z);
        }
#pragma unroll
        for (int s = 0; s < kMaxSplit; ++s) {
          // (a part at the maximum weighs 1, also where that is infinite: a sink of -inf or +inf)
          if (st[s].y != 0.f) weight[s] = st[s].x == top ? 1.f : ex2(st[s].x - top);
          sum = fmaf(st[s].y, weight[s], sum);
        }
        const bool live = sum > 0.f;
        const float inv = live ? (kFp8 ? v_ref * 0.015625f / sum : 1.0f / sum) : 0.f;
        __nv_bfloat16* orow = p.o + (int64_t)batch * p.o_sb + (int64_t)head * p.o_sh + (int64_t)q_row * p.o_ss;
        uint4* o4 = reinterpret_cast<uint4*>(orow);
        uint4* peer4 = p.o_peer.ptrs ? reinterpret_cast<uint4*>(peer_row(p.o_peer, batch, head, q_row)) : nullptr;
        for (int c = rank; c * 8 < p.d_v; c += p.n_split) {  // eight columns at a time, shared out over the cluster
          float4 x = make_float4(0.f, 0.f, 0.f, 0.f), y = x;
#pragma unroll
          for (int s = 0; s < kMaxSplit; ++s) {
            if (s >= p.n_split) break;
            const float4 u = cluster_ld_v4(cluster_addr(part + (2 * c) * 2 * kTile, s));
            const float4 w = cluster_ld_v4(cluster_addr(part + (2 * c + 1) * 2 * kTile, s));
            x.x = fmaf(u.x, weight[s], x.x), x.y = fmaf(u.y, weight[s], x.y);
            x.z = fmaf(u.z, weight[s], x.z), x.w = fmaf(u.w, weight[s], x.w);
            y.x = fmaf(w.x, weight[s], y.x), y.y = fmaf(w.y, weight[s], y.y);
            y.z = fmaf(w.z, weight[s], y.z), y.w = fmaf(w.w, weight[s], y.w);
          }
          const uint4 w = make_uint4(pack_bf16(x.x * inv, x.y * inv), pack_bf16(x.z * inv, x.w * inv),
                                     pack_bf16(y.x * inv, y.y * inv), pack_bf16(y.z * inv, y.w * inv));
          o4[c] = w;
          if (peer4) peer4[c] = w;
        }
        if (rank == 0) store_row_stats<kFp8, kSoftCap>(p, batch, head, q_row, live, top, sum, m_all, sink2, fixed_max);
      }
    } else if (ok && valid) {
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
        store_rows32_peer(row0, p.o_ss, p.o_peer, batch, head, q_row - lane, v, inv, g * 32, p.d_v);
      }
      store_row_stats<kFp8, kSoftCap>(p, batch, head, q_row, live, m_used, l, m_true, sink2, fixed_max);
    }
    tc_fence_before();  // O has been read, ahead of the next row's P
    if (kSplit) break;
    }
  }

  // ---- teardown
  if constexpr (kSplit) {
    if (warp >= 8) cluster_sync();  // the parts are in place
    cluster_sync();                 // they have been read
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 9) {
    __syncwarp();
    tmem_dealloc(tmem, 512);
  }
}

// ------------------------------------------------------------------------------------------
// host launcher
// ------------------------------------------------------------------------------------------
using FwdKernel = void (*)(CUtensorMap, CUtensorMap, CUtensorMap, FwdParams);
static FwdKernel fwd_kernel(bool split, int variant) {
  static const FwdKernel kernels[2][4] = {
      {splash_fwd_kernel<false, false, false, false>, splash_fwd_kernel<true, false, false, false>,
       splash_fwd_kernel<false, true, false, false>, splash_fwd_kernel<true, false, true, false>},
      {splash_fwd_kernel<false, false, false, true>, splash_fwd_kernel<true, false, false, true>,
       splash_fwd_kernel<false, true, false, true>, splash_fwd_kernel<true, false, true, true>}};
  return kernels[split][variant];
}

// CTAs that share a schedule row (256 query rows) of this call; the 128-wide kernels only
static int fwd_split(const SplashFwdArgs& a, const SplashShards& shards, int variant, const int32_t* clusters) {
  const int64_t q_shards = shards.q_shards > 1 ? shards.q_shards : 1;
  if (a.q_segment_ids != nullptr || (a.q_sequence != nullptr && q_shards == 1)) return 1;
  const int64_t n_rows = (a.q.size[2] / kTile * q_shards + 1) / 2;
  const RowWork rw = estimate_row_work(a.mask_fn, (int)n_rows, 2 * kTile, (int)(a.k.size[2] / kTile),
                                       n_rows * a.q.size[0] * a.q.size[1] * (shards.head_shards > 1 ? shards.head_shards : 1));
  return row_parts(rw, clusters, [&] {
    return cluster_capacity((const void*)fwd_kernel(true, variant), variant, kFwdThreads,
                            fwd_smem_bytes(variant & 1, variant == 3, true));
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
  const FwdKernel kernel = fwd_kernel(split, variant);
  const int smem = fwd_smem_bytes(fp8, p16, split);
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
