"""Grids that hold several tiles for every SM.

The CTAs of the kernels take over one tile after the other (operand rings, barrier phases and TMEM carry on
from tile to tile), so a call that fills the chip several times takes other paths than the small calls the
oracle is compared with.  Every head of such a call must get the bits of a call on that head alone.
"""
import math

import numpy as np
import pytest
import torch

from oracle import attention_ref
from tokamax_b200 import _native
from tokamax_b200 import fp8
from tokamax_b200 import splash_attention_kernel as splash
from tokamax_b200 import splash_attention_mask as mask_lib

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


def _run(kernel, q, k, v, do, seg, scale):
  q, k, v = (t.detach().requires_grad_(True) for t in (q, k, v))
  out, res = kernel(q, k, v, seg, logits_scale=scale)
  dq, dk, dv = torch.autograd.grad(out, (q, k, v), do)
  return {"out": out.detach(), "lse": res["logsumexp"], "dq": dq, "dk": dk, "dv": dv}


def _mask(kind, s):
  if kind == "window":
    return mask_lib.LocalMask((s, s), (300, 0), 0)
  if kind == "table":  # rows of tiles without a live block among them
    m = np.tril(np.ones((s, s), np.bool_))
    m[512:768] = False
    m[:, 640:896] = False
    return mask_lib.NumpyMask(m)
  return mask_lib.CausalMask((s, s))


# 13 tiles of 22 (batch, kv head) pairs: 286 CTAs and more for at most 148 SMs; an odd number of steps in rings of
# two, three and four slots
@pytest.mark.parametrize("d_qk,d_v", [(192, 128), (256, 256), (160, 160), (64, 192), (256, 72), (136, 200)])
@pytest.mark.parametrize("kind,soft_cap,segments", [("causal", None, False), ("window", 20.0, True), ("table", None, False)])
def test_heads_above_128_of_a_large_call_are_those_of_small_calls(d_qk, d_v, kind, soft_cap, segments):
  b, hkv, group, s = 2, 11, 2, 1664
  g = torch.Generator(device=DEV).manual_seed(d_qk + 3 * d_v)
  mk = lambda h, d: torch.randn(b, h, s, d, generator=g, device=DEV).to(torch.bfloat16)
  q, k, v, do = mk(hkv * group, d_qk), mk(hkv, d_qk), mk(hkv, d_v), mk(hkv * group, d_v)
  seg = None
  if segments:
    ids = torch.zeros((b, s), dtype=torch.int32, device=DEV)
    ids[0, 700:], ids[1, 130:], ids[1, 1500:] = 1, 1, 2
    seg = splash.SegmentIds(q=ids, kv=ids)
  config = splash.SplashConfig.get_default()
  if soft_cap:
    config = splash.dataclasses.replace(config, attn_logits_soft_cap=soft_cap)
  kernel = splash.make_splash_mha(_mask(kind, s), config=config, q_seq_shards=1, save_residuals=True)
  scale = 1 / math.sqrt(d_qk)
  whole = _run(kernel, q, k, v, do, seg, scale)
  kernel.check_errors()
  for h in range(0, hkv, 5):
    heads = slice(h * group, (h + 1) * group)
    part = _run(kernel, q[:, heads].contiguous(), k[:, h:h + 1].contiguous(), v[:, h:h + 1].contiguous(),
                do[:, heads].contiguous(), seg, scale)
    kernel.check_errors()
    for name in part:
      mine = whole[name][:, heads if name in ("out", "lse", "dq") else slice(h, h + 1)]
      assert torch.equal(mine, part[name]), (name, h)


# 7 schedule rows of 44 (batch, q head) pairs; the second tile of every head's last row does not exist
@pytest.mark.parametrize("d", [128, 64, 80])
@pytest.mark.parametrize("kind,soft_cap,segments,sinks", [("causal", None, False, True), ("window", 20.0, True, False),
                                                          ("table", None, False, False)])
def test_heads_up_to_128_of_a_large_call_are_those_of_its_shares(d, kind, soft_cap, segments, sinks):
  b, hkv, group, s = 2, 11, 2, 1664
  g = torch.Generator(device=DEV).manual_seed(d)
  mk = lambda h: torch.randn(b, h, s, d, generator=g, device=DEV).to(torch.bfloat16)
  q, k, v, do = mk(hkv * group), mk(hkv), mk(hkv), mk(hkv * group)
  seg = None
  if segments:
    ids = torch.zeros((b, s), dtype=torch.int32, device=DEV)
    ids[0, 700:], ids[1, 130:], ids[1, 1500:] = 1, 1, 2
    seg = splash.SegmentIds(q=ids, kv=ids)
  config = splash.SplashConfig.get_default()
  if soft_cap:
    config = splash.dataclasses.replace(config, attn_logits_soft_cap=soft_cap)
  kernel = splash.make_splash_mha(_mask(kind, s), config=config, q_seq_shards=1, save_residuals=True, repeatable_dq=True)
  sink = torch.randn(hkv * group, generator=g, device=DEV) if sinks else None
  scale = 1 / math.sqrt(d)

  def run(kern, q, k, v, do, sink):
    q, k, v = (t.detach().requires_grad_(True) for t in (q, k, v))
    out, res = kern(q, k, v, seg, sink, logits_scale=scale)
    dq, dk, dv = torch.autograd.grad(out, (q, k, v), do)
    return {"out": out.detach(), "lse": res["logsumexp"], "max": res["max_logits"], "dq": dq, "dk": dk, "dv": dv}

  whole = run(kernel, q, k, v, do, sink)
  kernel.check_errors()
  share = kernel.head_shard(hkv)  # cut as the whole call is, whatever its size
  for h in range(0, hkv, 5):
    heads = slice(h * group, (h + 1) * group)
    part = run(share, q[:, heads].contiguous(), k[:, h:h + 1].contiguous(), v[:, h:h + 1].contiguous(),
               do[:, heads].contiguous(), sink[heads] if sinks else None)
    share.check_errors()
    for name in part:
      mine = whole[name][:, slice(h, h + 1) if name in ("dk", "dv") else heads]
      assert torch.equal(mine, part[name]), (name, h)


# 13 kv tiles of 24 (batch, kv head) pairs: 312 CTAs, two tiles and more for an SM, with a soft cap too.  The two forms of
# the backward compute dk and dv by the same products in the same order; dq's are summed in another one.
@pytest.mark.parametrize("d_qk,d_v", [(128, 128), (64, 64), (80, 128), (128, 64)])
@pytest.mark.parametrize("kind,soft_cap,segments", [("causal", None, False), ("window", 20.0, True), ("window", None, True),
                                                    ("table", None, False), ("full", None, False)])
def test_both_backward_forms_of_a_large_call(d_qk, d_v, kind, soft_cap, segments):
  b, hkv, group, s = 2, 12, 2, 1664
  g = torch.Generator(device=DEV).manual_seed(d_qk + d_v)
  mk = lambda h, d: torch.randn(b, h, s, d, generator=g, device=DEV).to(torch.bfloat16)
  q, k, v, do = mk(hkv * group, d_qk), mk(hkv, d_qk), mk(hkv, d_v), mk(hkv * group, d_v)
  seg = None
  if segments:  # the second row's queries see no key of its last 164 tokens: kv tiles with steps that come to nothing
    ids = torch.zeros((b, s), dtype=torch.int32, device=DEV)
    ids[0, 700:], ids[1, 130:], ids[1, 1500:] = 1, 1, 2
    seg = splash.SegmentIds(q=ids.clamp(max=1) if kind == "window" else ids, kv=ids)
  config = splash.dataclasses.replace(splash.SplashConfig.get_default(), attn_logits_soft_cap=soft_cap)
  mask = mask_lib.FullMask((s, s)) if kind == "full" else _mask(kind, s)
  fused, split = (_run(splash.make_splash_mha(mask, config=config, q_seq_shards=1, save_residuals=True, repeatable_dq=r),
                       q, k, v, do, seg, 1 / math.sqrt(d_qk)) for r in (False, True))
  for name in ("out", "lse", "dk", "dv"):
    assert torch.equal(fused[name], split[name]), name
  # fp32 sums of the same products in another order, rounded to bf16 where they differ in the last bits
  assert ((fused["dq"].float() - split["dq"].float()).norm() / split["dq"].float().norm()).item() <= 1e-3


@pytest.mark.parametrize("p_format", ["e4m3", "f16"])
def test_e4m3_heads_of_a_large_call_are_those_of_its_shares(p_format):
  b, hkv, group, s = 2, 11, 2, 1664
  g = torch.Generator(device=DEV).manual_seed(3)
  mk = lambda h: torch.randn(b, h, s, 128, generator=g, device=DEV).to(torch.bfloat16)
  q, k, v = mk(hkv * group), mk(hkv), mk(hkv)
  kernel = splash.make_splash_mha(_mask("causal", s), q_seq_shards=1)
  run = lambda kern, *t: fp8.splash_fwd_fp8(kern, *(fp8.quantize_e4m3(x) for x in t), logits_scale=0.09, p_format=p_format)
  whole = run(kernel, q, k, v)
  for h in range(0, hkv, 5):
    heads = slice(h * group, (h + 1) * group)
    part = run(kernel.head_shard(hkv), q[:, heads].contiguous(), k[:, h:h + 1].contiguous(), v[:, h:h + 1].contiguous())
    kernel.check_errors()
    assert torch.equal(whole[:, heads], part), h


def _pairs_with_a_dead_tile(s):
  """A causal table that leaves out one tile of the pairs of a schedule row (256 query rows), or none.

  The warps of a tile that is dead in several of a CTA's rows have nothing to do in them, and may be rows behind the
  others when the tile is live again.  The last pair's second tile does not exist (its row is then empty).
  """
  m = np.tril(np.ones((s, s), np.bool_))
  for pair, dead in enumerate((1, 1, 0, 1, None, 1, 0)):
    if dead is not None:
      m[pair * 256 + dead * 128:pair * 256 + dead * 128 + 128] = False
  return m


# eight rows a CTA and more.  q_len 128: no row has its second tile
@pytest.mark.parametrize("variant", ["bf16", "soft_cap", "e4m3", "f16"])
@pytest.mark.parametrize("q_len,kv_len", [(1664, 1664), (128, 128), (128, 640)])
def test_rows_with_a_dead_tile_of_a_large_call(variant, q_len, kv_len):
  b, hkv, group = (2, 11, 8) if q_len > 128 else (8, 20, 8)
  g = torch.Generator(device=DEV).manual_seed(q_len + kv_len)
  mk = lambda h, s: torch.randn(b, h, s, 128, generator=g, device=DEV).to(torch.bfloat16)
  q, k, v = mk(hkv * group, q_len), mk(hkv, kv_len), mk(hkv, kv_len)
  dense = _pairs_with_a_dead_tile(q_len) if q_len > 128 else np.tril(np.ones((q_len, kv_len), np.bool_), kv_len - q_len)
  cap = 20.0 if variant == "soft_cap" else None
  config = splash.dataclasses.replace(splash.SplashConfig.get_default(), attn_logits_soft_cap=cap)
  kernel = splash.make_splash_mha(mask_lib.NumpyMask(dense), config=config, q_seq_shards=1,
                                  save_residuals=variant in ("bf16", "soft_cap"))
  scale = 1 / math.sqrt(128)

  def run(kern, q, k, v):
    if variant in ("e4m3", "f16"):
      t = fp8.splash_fwd_fp8(kern, *(fp8.quantize_e4m3(x) for x in (q, k, v)), logits_scale=scale, p_format=variant)
      return {"out": t}
    with torch.no_grad():
      out, res = kern(q, k, v, logits_scale=scale)
    return {"out": out, "lse": res["logsumexp"], "max": res["max_logits"]}

  whole = run(kernel, q, k, v)
  kernel.check_errors()
  share = kernel.head_shard(hkv)
  for h in range(0, hkv, 5):
    heads = slice(h * group, (h + 1) * group)
    part = run(share, q[:, heads].contiguous(), k[:, h:h + 1].contiguous(), v[:, h:h + 1].contiguous())
    share.check_errors()
    for name in part:
      assert torch.equal(whole[name][:, heads], part[name]), (name, h)
  live = torch.from_numpy(dense.any(1))
  assert not whole["out"][:, :, ~live].any()
  if "lse" not in whole:
    return
  for at, h in ((0, 3), (b - 1, hkv * group - 1)):
    kv = slice(h // group, h // group + 1)
    ro, rlse, rmax = attention_ref.attention_reference(q[at, h:h + 1].cpu(), k[at, kv].cpu(), v[at, kv].cpu(), dense, scale=scale,
                                                       attn_logits_soft_cap=cap)
    # P and the output are rounded to 8 bits, half an ulp (2^-9) each: at most 2^-8 of the largest |v| of a row's keys
    bound = 2.0 ** -8 * v[at, kv].float().abs().max().item()
    assert (whole["out"][at, h].float().cpu() - ro[0])[live].abs().max().item() <= bound
    assert (whole["lse"][at, h].cpu() - rlse[0])[live].abs().max().item() <= 1e-4  # fp32 sums of up to 1664 terms
    assert (whole["max"][at, h].cpu() - rmax[0])[live].abs().max().item() <= 1e-4


@pytest.mark.parametrize("d_qk,d_v", [(256, 256), (192, 128), (128, 128)])
@pytest.mark.parametrize("raised", [False, True])
def test_the_largest_weight_of_a_row_is_not_rounded(d_qk, d_v, raised):
  # Every row sees key r of its last 128 keys' first half with logit 0 (base 2) and key r of the second half with logit
  # x < 8: under the maximum of the 128 the second weighs 1, under that of 64 keys the rounded 2^x.  `raised`: 128 keys
  # of logit -20 come before, so that the maximum in use rises there.
  n = 256 if raised else 128
  g = torch.Generator().manual_seed(d_qk)
  x = (0.5 + 7 * torch.rand(128, generator=g)).to(torch.bfloat16)
  r = torch.arange(128)
  dense = np.zeros((128, n), np.bool_)
  dense[r, n - 128 + r % 64] = dense[r, n - 64 + r % 64] = True
  dense[:, :n - 128] = True
  q, k, v = torch.zeros(1, 1, 128, d_qk), torch.zeros(1, 1, n, d_qk), torch.zeros(1, 1, n, d_v)
  q[..., 0], q[..., 1] = x.float(), 1.0
  k[0, 0, n - 64:, 0], k[0, 0, :n - 128, 1] = 1.0, -20.0
  v[0, 0, n - 64:] = 1.0
  kernel = splash.make_splash_mha(mask_lib.NumpyMask(dense), q_seq_shards=1)
  q, k, v = (t.to(DEV, torch.bfloat16) for t in (q, k, v))
  out = kernel(q, k, v, logits_scale=math.log(2.0)).double().cpu()[0, 0]
  kernel.check_errors()
  w = torch.exp2(x.double())
  exact = (w / (w + 1 + (n - 128) * 2.0 ** -20))[:, None]
  # the output's rounding (2^-9 of a value below 1, half that above 1/2), and fp32 arithmetic on logits up to 20
  assert (out - exact).abs().max().item() <= 2.0 ** -9 + 20 * 2.0 ** -23


# 286 tiles and more, as above.  A fixed maximum drops the exchange of maxima between the warpgroups; a sink is counted once
@pytest.mark.parametrize("d_qk,d_v", [(192, 128), (256, 256)])
@pytest.mark.parametrize("fixed,sinks", [(True, False), (True, True), (False, True)])
def test_heads_above_128_with_a_fixed_maximum_or_sinks_of_a_large_call(d_qk, d_v, fixed, sinks):
  b, hkv, group, s = 2, 11, 2, 1664
  g = torch.Generator(device=DEV).manual_seed(d_qk)
  mk = lambda h, d: torch.randn(b, h, s, d, generator=g, device=DEV).to(torch.bfloat16)
  q, k, v = mk(hkv * group, d_qk), mk(hkv, d_qk), mk(hkv, d_v)
  sink = torch.randn(hkv * group, generator=g, device=DEV) if sinks else None
  top = 6 + torch.rand(hkv * group, generator=g, device=DEV) if fixed else None
  kernel = splash.make_splash_mha(_mask("causal", s), q_seq_shards=1, save_residuals=True)

  def run(heads, q, k, v):
    with torch.no_grad():
      out, res = kernel(q, k, v, None, sink[heads] if sinks else None, max_logit_value=top[heads] if fixed else None,
                        logits_scale=1 / math.sqrt(d_qk))
    kernel.check_errors()
    return {"out": out, "lse": res["logsumexp"], "max": res["max_logits"]}

  whole = run(slice(None), q, k, v)
  for h in range(0, hkv, 5):
    heads = slice(h * group, (h + 1) * group)
    part = run(heads, q[:, heads].contiguous(), k[:, h:h + 1].contiguous(), v[:, h:h + 1].contiguous())
    for name in part:
      assert torch.equal(whole[name][:, heads], part[name]), (name, h)
  h = hkv * group - 1
  ro, rlse, _ = attention_ref.attention_reference(q[1, h:].cpu(), k[1, -1:].cpu(), v[1, -1:].cpu(), np.tril(np.ones((s, s), np.bool_)),
                                                  scale=1 / math.sqrt(d_qk), sinks=sink[h:].cpu() if sinks else None)
  # P and the output are rounded to 8 bits, half an ulp each
  assert (whole["out"][1, h].float().cpu() - ro[0]).abs().max().item() <= 2.0 ** -8 * v[1, -1].float().abs().max().item()
  assert (whole["lse"][1, h].cpu() - rlse[0]).abs().max().item() <= 1e-4


@pytest.mark.parametrize("d_qk,d_v", [(128, 128), (64, 64), (192, 128), (256, 256)])
def test_device_masks_of_a_large_call(d_qk, d_v):
  # schedules built on the device (an end for each row of each batch row) against the host's tables; the fused backward
  # up to 128, and its dq against the repeatable one
  b, hkv, group, s = 2, 11, 2, 1664
  g = torch.Generator(device=DEV).manual_seed(d_qk)
  mk = lambda h, d: torch.randn(b, h, s, d, generator=g, device=DEV).to(torch.bfloat16)
  q, k, v, do = mk(hkv * group, d_qk), mk(hkv, d_qk), mk(hkv, d_v), mk(hkv * group, d_v)
  dense = _pairs_with_a_dead_tile(s)
  dense[:, 300:900] &= np.random.default_rng(d_qk).random((s, 600)) < 0.5
  kernels = [splash.make_dynamic_splash_mha(torch.from_numpy(dense).to(DEV), save_residuals=True),
             splash.make_splash_mha(mask_lib.NumpyMask(dense), q_seq_shards=1, save_residuals=True),
             splash.make_splash_mha(mask_lib.NumpyMask(dense), q_seq_shards=1, save_residuals=True, repeatable_dq=True)]
  device, host, repeatable = (_run(kernel, q, k, v, do, None, 1 / math.sqrt(d_qk)) for kernel in kernels)
  for kernel in kernels:
    kernel.check_errors()
  for name in ("out", "lse", "dk", "dv") if d_qk <= 128 else device:
    assert torch.equal(device[name], host[name]), name
  for name in ("dq", "dk", "dv"):
    want = repeatable[name].float()
    # the same products summed in another order (fp32), rounded to bf16 where they differ in the last bits
    for other in (device, host):
      assert ((other[name].float() - want).norm() / want.norm()).item() <= 1e-3, name


def test_peer_outputs_of_a_large_call():
  # rows that CTAs take over, stored twice: in the call's own tensor and in the buffer of the rank that owns them
  b, hq, hkv, s, d, world, rank = 2, 44, 22, 1536, 128, 2, 1
  g = torch.Generator(device=DEV).manual_seed(5)
  mk = lambda h: torch.randn(b, h, s, d, generator=g, device=DEV).to(torch.bfloat16)
  q, k, v, do = mk(hq), mk(hkv), mk(hkv), mk(hq)
  kernel = splash.make_splash_mha(_mask("causal", s), q_seq_shards=1)
  s_loc = s // world

  def receive(heads):
    bufs = [torch.full((b, heads * world, s_loc, d), 7.0, dtype=torch.bfloat16, device=DEV) for _ in range(world)]
    ptrs = torch.tensor([t.data_ptr() for t in bufs], dtype=torch.int64, device=DEV)
    po = _native.SplashPeerOutput()
    po.ptrs, po.base_bytes, po.rows_per_peer = ptrs.data_ptr(), 0, s_loc
    po.stride_b, po.stride_h, po.stride_s, po.head0 = heads * world * s_loc * d, s_loc * d, d, rank * heads
    return bufs, ptrs, po

  recv = [receive(h) for h in (hq, hq, hkv, hkv)]
  _, _, _, o, lse, _, _ = splash.splash_forward(kernel, q, k, v, None, None, 0.09, None, None, 0, o_peer=recv[0][2])
  dq, dk, dv, _ = splash.splash_backward(kernel, q, k, v, o, lse, do, None, None, 0.09, 0, peers=tuple(r[2] for r in recv[1:]))
  kernel.check_errors()
  assert torch.equal(o, kernel(q, k, v, logits_scale=0.09))
  for (bufs, _, _), local, heads in zip(recv, (o, dq, dk, dv), (hq, hq, hkv, hkv)):
    for peer in range(world):
      assert torch.equal(bufs[peer][:, rank * heads:], local[:, :, peer * s_loc:(peer + 1) * s_loc])
      assert (bufs[peer][:, :rank * heads] == 7.0).all()
