"""attn_logits_soft_cap: logits = cap * tanh(scale * q k^T / cap), forward and backward.

Reference: splash_attention_kernel.py:202-296 (cap, then mask), base.py:92-94 and :159-163 (the
backward chain factor 1 - tanh^2).
"""
import dataclasses
import math

import numpy as np
import pytest
import torch

from oracle import attention_ref
from tokamax_b200 import splash_attention_kernel as splash
from tokamax_b200 import splash_attention_mask as mask_lib

pytestmark = pytest.mark.gpu
D = 128
DEV = "cuda:0"


def _rel(a, ref):
  return ((a.float().cpu() - ref).norm() / ref.norm().clamp_min(1e-20)).item()


@pytest.mark.parametrize("cap,scale,dims", [(30.0, 1 / math.sqrt(D), (D, D)), (8.0, 0.35, (D, D)),
                                            (2.0, 1 / math.sqrt(D), (D, D)), (8.0, 0.2, (192, 128)),
                                            (4.0, 1 / 16, (256, 256))])
@pytest.mark.parametrize("kind", ["causal", "local_segments"])
def test_soft_cap_forward_backward(cap, scale, dims, kind):
  """(128, 128), and the head dims above 128 that run kernels of their own."""
  b, hq, hkv, s = 1, 4, 2, 512
  d_qk, d_v = dims
  g = torch.Generator().manual_seed(int(cap * 10) + len(kind) + d_qk)
  mk = lambda *shape: torch.randn(*shape, generator=g).to(torch.bfloat16)
  q, k, v, do = mk(b, hq, s, d_qk), mk(b, hkv, s, d_qk), mk(b, hkv, s, d_v), mk(b, hq, s, d_v)
  seg = None
  if kind == "causal":
    mask = mask_lib.CausalMask((s, s))
  else:
    mask = mask_lib.LocalMask((s, s), (200, 0), 0)
    ids = torch.from_numpy(np.repeat(np.arange(4, dtype=np.int32), [100, 156, 56, 200]))
    seg = (ids, ids)
  dense = np.asarray(mask[:, :])
  cfg = dataclasses.replace(splash.SplashConfig.get_default(), attn_logits_soft_cap=cap)
  kernel = splash.make_splash_mha_single_device(mask, config=cfg, save_residuals=True)
  qd, kd, vd = (t.to(DEV).requires_grad_(True) for t in (q, k, v))
  seg_dev = None if seg is None else splash.SegmentIds(seg[0][None].to(DEV), seg[1][None].to(DEV))
  out, res = kernel(qd, kd, vd, seg_dev, logits_scale=scale)
  out.backward(do.to(DEV))
  kernel.check_errors()
  ro, rlse, rmx = attention_ref.attention_reference(q[0], k[0], v[0], dense, seg, scale=scale,
                                                    attn_logits_soft_cap=cap)
  rdq, rdk, rdv = attention_ref.attention_reference_vjp(do[0], q[0], k[0], v[0], dense, seg, ro.to(torch.bfloat16),
                                                        rlse, scale=scale, attn_logits_soft_cap=cap)
  assert ((out.float().cpu()[0] - ro).abs() <= 1e-2 + 4e-3 * ro.abs()).all()
  assert (res["logsumexp"].cpu()[0] - rlse).abs().max() <= 1e-3
  assert (res["max_logits"].cpu()[0] - rmx).abs().max() <= 1e-3
  assert (res["max_logits"] <= cap + 1e-4).all()
  for got, ref in ((qd.grad[0], rdq), (kd.grad[0], rdk), (vd.grad[0], rdv)):
    assert _rel(got, ref) <= 1e-2


# A warp whose arguments of tanh are all at most 1/2 takes a polynomial, any other the special functions.  A tile has warps of
# either kind here: queries grow in runs of 16 rows until the largest argument of a run lies at `top` and around it.  Of rows
# 0 and 64 .. the arguments are zero and tiny.
@pytest.mark.parametrize("repeatable", [False, True])
@pytest.mark.parametrize("d,kind", [(128, "full"), (128, "causal"), (64, "full"), (256, "full"), (192, "causal")])
@pytest.mark.parametrize("top", [0.49, 0.5, 0.51, 40.0])
def test_both_forms_of_tanh_in_one_tile(d, kind, top, repeatable):
  s, cap, scale = 256, 20.0, 1 / math.sqrt(d)
  g = torch.Generator().manual_seed(d)
  q, k, v, do = (torch.randn(1, 1, s, d, generator=g, dtype=torch.float64) for _ in range(4))
  largest = (q @ k.transpose(-1, -2)).abs().amax(-1, keepdim=True) * scale / cap
  grow = torch.tensor([0.0, 1e-4, 0.1, 0.5, 0.9, 1.0, 1.0, 1.2]).repeat_interleave(16).repeat(2).view(1, 1, s, 1)
  q, k, v, do = (t.to(torch.bfloat16) for t in (q / largest * top * grow, k, v, do))
  mask = mask_lib.FullMask((s, s)) if kind == "full" else mask_lib.CausalMask((s, s))
  dense = np.tril(np.ones((s, s), np.bool_)) if kind == "causal" else np.ones((s, s), np.bool_)
  cfg = dataclasses.replace(splash.SplashConfig.get_default(), attn_logits_soft_cap=cap)
  kernel = splash.make_splash_mha(mask, config=cfg, q_seq_shards=1, save_residuals=True, repeatable_dq=repeatable)
  ts = [t.to(DEV).requires_grad_(True) for t in (q, k, v)]
  out, res = kernel(*ts, logits_scale=scale)
  grads = torch.autograd.grad(out, ts, do.to(DEV))
  kernel.check_errors()
  wide = [t.double().requires_grad_(True) for t in (q, k, v)]
  x = cap * torch.tanh(wide[0] @ wide[1].transpose(-1, -2) * (scale / cap))
  x = x.masked_fill(~torch.from_numpy(dense), -math.inf)
  ro = torch.softmax(x, -1) @ wide[2]
  rgrads = torch.autograd.grad(ro, wide, do.double())
  # tanh to 1e-6 absolute times the cap, and fp32 sums of d products and of s weights
  bound = cap * 1e-6 + 1e-5
  assert (res["logsumexp"].cpu().double() - torch.logsumexp(x, -1)).abs().max().item() <= bound
  assert (res["max_logits"].cpu().double() - x.amax(-1)).abs().max().item() <= bound
  # P and the output are rounded to 8 bits, half an ulp (2^-9) each
  assert (out.cpu().double() - ro).abs().max().item() <= 2.0 ** -8 * v.double().abs().max().item()
  for got, want in zip(grads, rgrads):
    assert ((got.cpu().double() - want).norm() / want.norm()).item() <= 1e-2


# tanh is a function of its argument alone: the polynomial up to 1/2, the special functions above, whatever a row's neighbours
# and its masked keys hold.  The middle document shares tiles and warps with the others; once its arguments are tiny, once
# they run far beyond 1/2, its products with the other documents' tokens too.
@pytest.mark.parametrize("repeatable", [False, True])
@pytest.mark.parametrize("dims", [(64, 64), (80, 80), (128, 128), (192, 128), (256, 256)])
@pytest.mark.parametrize("kind", ["full", "causal"])
def test_a_documents_bits_do_not_depend_on_its_neighbours(kind, dims, repeatable):
  s, cap, ends = 256, 20.0, (48, 200, 256)
  d_qk, d_v = dims
  g = torch.Generator().manual_seed(d_qk)
  q, k, v, do = (torch.randn(1, 2, s, d, generator=g) for d in (d_qk, d_qk, d_v, d_v))
  ids = torch.repeat_interleave(torch.arange(3, dtype=torch.int32), torch.tensor([ends[0], ends[1] - ends[0], s - ends[1]]))
  mask = mask_lib.FullMask((s, s)) if kind == "full" else mask_lib.CausalMask((s, s))
  cfg = dataclasses.replace(splash.SplashConfig.get_default(), attn_logits_soft_cap=cap)
  kernel = splash.make_splash_mha(mask, config=cfg, q_seq_shards=1, save_residuals=True, repeatable_dq=repeatable)

  def run(factor):
    grow = torch.ones(s, 1)
    grow[ends[0]:ends[1]] = factor
    qd, kd, vd, dod = (t.to(torch.bfloat16).to(DEV) for t in (q * grow, k * grow, v, do))
    ts = [t.requires_grad_(True) for t in (qd, kd, vd)]
    seg = splash.SegmentIds(ids[None].to(DEV), ids[None].to(DEV))
    out, res = kernel(*ts, seg, logits_scale=1 / math.sqrt(d_qk))
    grads = torch.autograd.grad(out, ts, dod)
    kernel.check_errors()
    return (out, res["logsumexp"][..., None], res["max_logits"][..., None], *grads)

  small, large = run(0.01), run(30.0)
  for name, a, b in zip(("out", "lse", "max", "dq", "dk", "dv"), small, large):
    for rows in (slice(0, ends[0]), slice(ends[1], s)):
      assert torch.equal(a[:, :, rows], b[:, :, rows]), name
    assert not torch.equal(a, b)


def test_soft_cap_changes_the_result_and_rejects_bad_values():
  s = 256
  g = torch.Generator().manual_seed(3)
  q = torch.randn(1, 2, s, D, generator=g).to(torch.bfloat16).to(DEV)
  mask = mask_lib.CausalMask((s, s))
  plain = splash.make_splash_mha_single_device(mask)(q, q, q, logits_scale=0.3)
  cfg = dataclasses.replace(splash.SplashConfig.get_default(), attn_logits_soft_cap=3.0)
  capped = splash.make_splash_mha_single_device(mask, config=cfg)(q, q, q, logits_scale=0.3)
  assert (plain.float() - capped.float()).abs().max() > 0.05
  bad = dataclasses.replace(splash.SplashConfig.get_default(), attn_logits_soft_cap=-1.0)
  with pytest.raises(ValueError):
    splash.make_splash_mha_single_device(mask, config=bad)(q, q, q)
