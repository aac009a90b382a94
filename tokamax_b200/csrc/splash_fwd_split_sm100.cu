// The forward for head dims up to 128 where the grid leaves SMs idle: a cluster of CTAs shares each schedule row.
//
// A CTA is the whole-row forward's of splash_fwd_sm100.cu (roles, TMEM, rings) on its part of one row's kv tiles, as if
// the row held nothing else; it has no other row.  Afterwards every CTA leaves its O (fp32), maximum and sum in its
// own shared memory (the ring is free by then), and the cluster adds them up over distributed shared
// memory, each CTA a share of the columns: no scratch in global memory, no second launch, and the
// order of the additions is fixed.  split_for() (splash_split.cuh) holds the rule.
//
// A kernel of its own beside the whole rows', whose loop over rows it does not need: as one kernel with that loop
// compiled out, 512 query rows of 32 heads against 16384 keys took 130.8 us instead of 127.4 (head dim 128), or 116.8
// instead of 114.3 (64), by the form of the source that was common to both.
#include "splash_fwd_steps.cuh"

namespace sb {

struct SplitBarriers {
  uint64_t q_full[2];
  uint64_t kv_full[kFwdStages];
  uint64_t kv_empty[kFwdStages];
  uint64_t s_full[2];
  uint64_t p_half[2];    // the first 64 key columns of P are in TMEM (the first half of the p v MMAs may go)
  uint64_t p_full[2];
  uint64_t o_done[2];
  uint64_t vc_full[2];   // e4m3 with f16 P: a V tile has been converted to f16
  uint64_t vc_empty[2];  //                  the p v MMAs that read it have completed
  uint32_t tmem_base;
  uint32_t abort_flag;
  uint32_t early_exit;
};

// a CTA's part of the result lies over the operand tiles: 32 x 256 words of 16 bytes, one more row of statistics
constexpr int kPartBytes = (kHeadDim / 4 + 1) * 2 * kTile * 16;
__host__ __device__ constexpr int split_operand_bytes(bool fp8, bool p16) {
  return fwd_operand_bytes(fp8, p16) < kPartBytes ? kPartBytes : fwd_operand_bytes(fp8, p16);
}
int fwd_split_smem_bytes(int variant) {
  return split_operand_bytes(variant & 1, variant == 3) + 1024 /*barriers*/ + 1024 /*alignment slack*/;
}

template <bool kFp8, bool kSoftCap, bool kP16>
__global__ void __launch_bounds__(kFwdThreads, 1)
splash_fwd_split_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                        const __grid_constant__ CUtensorMap tm_v, const FwdParams p) {
  constexpr int kTB = kFp8 ? kFp8TileBytes : kTileBytes;  // bytes of one operand tile
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  uint8_t* q_smem = smem;                                  // 2 tiles
  static_assert(!kP16 || kFp8, "the f16-P variant is a variant of the e4m3 forward");
  uint8_t* kv_smem = smem + 2 * kTB;                       // ring
  uint8_t* vc_smem = smem + (2 + kFwdStages) * kTB;        // kP16: two f16 images of V tiles
  SplitBarriers* bars = reinterpret_cast<SplitBarriers*>(smem + split_operand_bytes(kFp8, kP16));

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const unsigned rank = cluster_rank();
  const CtaWork work = cta_work_at(blockIdx.x / p.n_split, p.row_order, p.n_rows, p.n_groups, p.chunk_groups, true);
  const int row = work.row;
  const int head = work.group % p.q_heads;
  const int batch = work.group / p.q_heads;
  const int kv_head = head / (p.q_heads / p.kv_heads);
  const int ebeg = p.row_ptr[row];
  const int eend = p.row_end ? p.row_end[(int64_t)batch * p.n_rows + row] : p.row_ptr[row + 1];
  const int4* entries = p.entries + (int64_t)batch * p.entries_per_batch;
  const PartWalk<true> walk(entries, ebeg, eend, p.n_split);  // the entries of this CTA
  const int efirst = walk.first(walk.offset((int)rank));
  const int qt0 = row * 2;

  if (threadIdx.x == 0) {
    bars->early_exit = *reinterpret_cast<volatile uint32_t*>(p.err);
    bars->abort_flag = bars->early_exit;  // (read by the other CTAs of the cluster)
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
    mbar_fence_init();
  }
  __syncthreads();
  if (bars->early_exit != 0) {  // an earlier CTA already reported a fault
    cluster_sync();  // the others may not have seen it: no CTA leaves while its shared memory may be read
    cluster_sync();
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
      for (int e = efirst; e < eend; e = walk.next(e), ++n) {
        const uint32_t it = 2 * n + 1, s = it % kFwdStages, j = n & 1u;
        bool ok = mbar_wait(&bars->kv_full[s], (it / kFwdStages) & 1u, ab, 0x600u + s);
        if (ok) ok = mbar_wait(&bars->vc_empty[j], ((n >> 1) & 1u) ^ 1u, ab, 0x610u + j);
        if (!__all_sync(0xffffffffu, ok)) break;
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
    }
   } else if (warp == 8) {
    // ------------------------------------------------------------------ TMA producer
    if (elect_one()) {
      tma_prefetch_desc(&tm_q);
      tma_prefetch_desc(&tm_k);
      tma_prefetch_desc(&tm_v);
      for (int i = 0; i < 2; ++i) {
        if (qt0 + i < p.n_q_tiles) {
          uint8_t* dst = q_smem + i * kTB;
          const bool two = !kFp8 && p.d_qk > 64;  // bf16 tiles are two 64-column halves
          mbar_arrive_expect_tx(&bars->q_full[i], (kFp8 || two) ? kTB : kHalfBytes);
          tma_load_4d(dst, &tm_q, &bars->q_full[i], 0, (qt0 + i) * kTile, head, batch);
          if (two) tma_load_4d(dst + kHalfBytes, &tm_q, &bars->q_full[i], 64, (qt0 + i) * kTile, head, batch);
        }
      }
      uint32_t it = 0;
      bool ok = true;
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
      bool ok = true;
      for (int i = 0; i < 2 && ok; ++i)
        if (qt0 + i < p.n_q_tiles) ok = mbar_wait(&bars->q_full[i], 0, ab, 0x200u + i);

      auto issue_qk = [&](int i, uint32_t slot) {
        fwd_issue_qk<kFp8>(tmem + i * kTile, q_addr + i * kTB, kv_addr + slot * kTB, p.nk_qk);
        tc_commit(&bars->s_full[i]);
      };
      auto issue_pv = [&](int i, uint32_t slot, bool acc, int half) {
        fwd_issue_pv<kFp8, kP16>(tmem + 2 * kTile + i * kTile, tmem + i * kTile,
                                 kP16 ? vc_addr + slot * kTileBytes : kv_addr + slot * kTB, idesc_pv, acc, half);
      };

      int e = efirst;
      uint32_t pcnt[2] = {0, 0};
      bool started[2] = {false, false};
      if (efirst < eend && ok) {
        const int4 e0 = entries[efirst];
        ok = mbar_wait(&bars->kv_full[0], 0, ab, 0x300u);
        if (ok) {
          mma_issue_fence();
          for (int i = 0; i < 2; ++i)
            if ((e0.y >> (2 * i)) & 3) issue_qk(i, 0);
          tc_commit(&bars->kv_empty[0]);
        }
        int4 nxt = e0;
        for (int n = 0; e < eend && ok; ++n) {
          const int4 cur = nxt;
          e = walk.next(e);
          const bool has_next = e < eend;
          if (has_next) nxt = entries[e];
          const uint32_t itv = 2 * n + 1, itk = 2 * n + 2;
          const uint32_t vslot = itv % kFwdStages, kslot = itk % kFwdStages;
          const uint32_t vc = n & 1u;  // kP16: which f16 image holds this step's V
          if constexpr (kP16)
            ok = mbar_wait(&bars->vc_full[vc], (n >> 1) & 1u, ab, 0x340u + vc);
          else
            ok = mbar_wait(&bars->kv_full[vslot], (itv / kFwdStages) & 1u, ab, 0x310u + vslot);
          if (ok && has_next)
            ok = mbar_wait(&bars->kv_full[kslot], (itk / kFwdStages) & 1u, ab, 0x320u + kslot);
          if (!ok) break;
          mma_issue_fence();
          for (int i = 0; i < 2 && ok; ++i) {
            if ((cur.y >> (2 * i)) & 3) {
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
            if (has_next && ((nxt.y >> (2 * i)) & 3)) issue_qk(i, kslot);
          }
          if (ok && has_next) tc_commit(&bars->kv_empty[kslot]);
        }
      }
      tc_commit(&bars->o_done[0]);  // (the parts go over the operand tiles: not before both tiles' MMAs have read them)
      tc_commit(&bars->o_done[1]);
    }
   }
  } else {
    // ------------------------------------------------------------------ softmax warpgroups
    setmaxnreg_inc<kSoftmaxRegs>();
    const int i = warp >> 2;           // q tile within the pair
    const int wq = warp & 3;           // TMEM lane quarter this warp may touch
    const int r = wq * 32 + lane;      // row within the tile
    const int q_tile = qt0 + i;
    const bool valid = q_tile < p.n_q_tiles;
    const int q_row = valid ? q_tile * kTile + r : 0;
    const int qi = p.q_sequence ? p.q_sequence[q_row] : q_row;
    const RowInterval iv = mask_fn_interval(p.fn, qi);
    const bool has_seg = p.q_seg != nullptr;
    const int q_seg = has_seg ? p.q_seg[(int64_t)batch * p.q_len + q_row] : 0;
    const int32_t* kv_seg_row = has_seg ? p.kv_seg + (int64_t)batch * p.kv_len : nullptr;
    const uint32_t lane_addr = (uint32_t)(wq * 32) << 16;
    const uint32_t t_s = tmem + lane_addr + i * kTile;
    const uint32_t t_o = tmem + lane_addr + 2 * kTile + i * kTile;
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
    const bool fixed_max = p.max_logit_value != nullptr;
    float sink2 = -INFINITY;  // sink logit in log2 units
    if (p.sinks != nullptr) sink2 = p.sinks[head] * kLog2e;
    const bool own_sink = p.sinks != nullptr && rank == 0;  // one CTA of the cluster counts it
    if (fixed_max) {
      m_used = p.max_logit_value[head] * kLog2e;
      if (own_sink) l = ex2(sink2 - m_used);
    } else if (own_sink) {
      m_used = sink2;
      l = 1.f;
    }
    uint32_t cnt = 0;
    bool started = false;
    bool ok = true;

    int4 ent_next = efirst < eend ? entries[efirst] : make_int4(0, 0, 0, 0);
    float ks_next = 1.f, vs_next = 1.f;
    if constexpr (kFp8) {
      if (efirst < eend) {
        ks_next = __ldg(k_scale + ent_next.x);
        vs_next = __ldg(v_scale + ent_next.x);
      }
    }
    int e_last = 0, x_due = ent_next.x, e_probe = efirst;
    for (int e = efirst; e < eend; e = e_probe) {
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
      const int4 ent = ent_next;
      const float ks = ks_next, vs = vs_next;
      if (e_probe < eend) {  // fetched a step ahead of its use
        ent_next = entries[e_probe];
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
    if (ok) {
      ok = mbar_wait(&bars->o_done[i], 0, ab, 0x500u + i);
      ok = __all_sync(0xffffffffu, ok);
    }
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
  }

  // ---- teardown
  if (warp >= 8) cluster_sync();  // the parts are in place
  cluster_sync();                 // they have been read
  tc_fence_before();
  __syncthreads();
  if (warp == 9) {
    __syncwarp();
    drain_after_give_up(&bars->abort_flag);
    tmem_dealloc(tmem, 512);
  }
}

FwdKernel fwd_split_kernel(int variant) {
  static const FwdKernel kernels[4] = {splash_fwd_split_kernel<false, false, false>, splash_fwd_split_kernel<true, false, false>,
                                       splash_fwd_split_kernel<false, true, false>, splash_fwd_split_kernel<true, false, true>};
  return kernels[variant];
}

}  // namespace sb
