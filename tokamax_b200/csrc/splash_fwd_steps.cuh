// What the two forwards for head dims up to 128 have in common: a CTA's rows left whole (splash_fwd_sm100.cu) and rows
// shared by a cluster (splash_fwd_split_sm100.cu).
#pragma once

#include "splash_fwd_params.cuh"

namespace sb {

// Variants: 0 bf16, 1 e4m3, 2 bf16 with a soft cap, 3 e4m3 with f16 P.
using FwdKernel = void (*)(CUtensorMap, CUtensorMap, CUtensorMap, FwdParams);
FwdKernel fwd_split_kernel(int variant);  // rows shared by a cluster
int fwd_split_smem_bytes(int variant);

// Q of two tiles, the ring of K and V, f16 images of two V tiles
__host__ __device__ constexpr int fwd_operand_bytes(bool fp8, bool p16) {
  return (2 + kFwdStages) * (fp8 ? kFp8TileBytes : kTileBytes) + (p16 ? 2 * kTileBytes : 0);
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


// S_i = Q_i K^T : both operands K-major.  bf16: eight K=16 slices across two swizzle halves; e4m3: four K=32 slices
// inside the single 128-byte-wide tile.
template <bool kFp8>
__device__ __forceinline__ void fwd_issue_qk(uint32_t t_s, uint32_t a0, uint32_t b0, int nk_qk) {
  constexpr uint32_t idesc =
      kFp8 ? make_idesc_e4m3(kTile, kTile, false, false) : make_idesc_bf16(kTile, kTile, false, false);
  const SmemDesc da = make_smem_desc_sw128(a0, 16, 1024), db = make_smem_desc_sw128(b0, 16, 1024);
  if constexpr (kFp8) {
#pragma unroll
    for (int k = 0; k < 4; ++k) umma_ss_f8(t_s, desc_at(da, k * 32), desc_at(db, k * 32), idesc, k > 0 ? 1u : 0u);
  } else {
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      // head dims below 128: the remaining slices multiply zeros (nk_qk == 8 is tested first so
      // that the full-width path stays a straight run of eight MMAs)
      if (nk_qk != 8 && k >= nk_qk) break;
      const uint32_t off = (k >> 2) * kHalfBytes + (k & 3) * 32;
      umma_ss(t_s, desc_at(da, off), desc_at(db, off), idesc, k > 0 ? 1u : 0u);
    }
  }
}

// Instruction descriptor of p v.  N: the output's columns, 128, or 64 when v has at most 64 (half the MMA work; the V
// tile's second half is then neither loaded nor read).  (kind::f16 with format code 0 for A and B is f16 x f16: the same
// bits as the e4m3 descriptor.)
template <bool kFp8>
__device__ __forceinline__ uint32_t fwd_idesc_pv(int d_v) {
  return kFp8 ? make_idesc_e4m3(kTile, kHeadDim, false, true)
              : make_idesc_bf16(kTile, (!kFp8 && d_v <= 64) ? 64 : kHeadDim, false, true);
}

// O_i (+)= P_i V : A from TMEM, B = V tile read MN-major (head_dim contiguous): 8 kv rows x 128 B per core group
// (SBO 1024).  bf16: 64-column halves 16 KiB apart (LBO), K=16 slices 2 KiB apart; e4m3: the 128 columns fit one
// 128-byte row, K=32 slices 4 KiB apart, P packed four values per TMEM column.
// `half` 0 / 1: the K slices over the first / last 64 key columns of P (the softmax warps hand P over in two halves, so
// that the first MMAs run while the second half is still being made)
template <bool kFp8, bool kP16>
__device__ __forceinline__ void fwd_issue_pv(uint32_t t_o, uint32_t t_p, uint32_t b0, uint32_t idesc, bool acc, int half) {
  if constexpr (kFp8 && !kP16) {
    const SmemDesc db = make_smem_desc_sw128(b0, 16, 1024);
#pragma unroll
    for (int kk = 0; kk < 2; ++kk) {
      const int k = half * 2 + kk;
      umma_ts_f8(t_o, t_p + k * 8, desc_at(db, k * 4096), idesc, (acc || k > 0) ? 1u : 0u);
    }
  } else {
    const SmemDesc db = make_smem_desc_sw128(b0, kHalfBytes, 1024);
#pragma unroll
    for (int kk = 0; kk < 4; ++kk) {
      const int k = half * 4 + kk;
      umma_ts(t_o, t_p + k * 8, desc_at(db, k * 2048), idesc, (acc || k > 0) ? 1u : 0u);
    }
  }
}

// Softmax of one 128 x 128 score tile, a thread a row: masks it, raises the maximum in use where it has to (O is then
// rescaled), writes P over the scores and hands it to the MMAs in two halves.  The scores are in TMEM.
template <bool kFp8, bool kSoftCap, bool kP16>
__device__ __forceinline__ void fwd_softmax_step(const FwdParams& p, uint64_t* p_half, uint64_t* p_full, uint32_t t_s,
                                                 uint32_t t_o, int i, int lane, const int4& ent, int st, float c, float v_share,
                                                 float log_share, const RowInterval& iv, int q_row, bool has_seg, int q_seg,
                                                 const int32_t* kv_seg_row, bool fixed_max, bool started, float& m_used,
                                                 float& m_true, float& l) {
  // e4m3 P must stay below 448; f16 P (times 2^6) below 65504; bf16 P has the range of fp32
  constexpr float kThreshold = (kFp8 && !kP16) ? kFp8RescaleThreshold : kRescaleThreshold;
  // e4m3: P * 2^shift * r with r = v scale / largest v scale in (0, 1]; it and its logarithm come from the caller, which works
  // them out ahead of the wait for the scores (behind it: 32768 keys 13.04 -> 12.93 ms, f16 P 2 x 8192 952 -> 933 us)
  const float r = v_share;
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
    tanh_all(s, p.softcap_a);
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
    const float m_sub = m_used - kFp8PShift - log_share;
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
        if (lane == 0) mbar_arrive(p_half);
      }
    }
    l += (ls0 + ls1) * __fdividef(0.015625f, r);
  } else if constexpr (kFp8) {
    // P * 2^shift * r, see above
    const float m_sub = m_used - kFp8PShift - log_share;
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
        if (lane == 0) mbar_arrive(p_half);
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
        if (lane == 0) mbar_arrive(p_half);
      }
    }
    ls0 = lsa.x + lsb.x;
    ls1 = lsa.y + lsb.y;
    l += ls0 + ls1;
  }
  tmem_st_wait();
  tc_fence_before();
  __syncwarp();
  if (lane == 0) mbar_arrive(p_full);
}

}  // namespace sb
