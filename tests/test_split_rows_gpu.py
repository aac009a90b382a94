"""Grids that leave SMs idle: schedule rows shared by a cluster of CTAs, against the CPU oracle.

Few heads, and rows that are shared where the test says so: every way of forming a row's entries (causal
offset, window, chunks, table mask; segment ids, whose rows stay whole), odd numbers of query tiles, parts
of unequal length, rows without a live key in some part, sinks (counted once) and a fixed maximum; every
number of parts, 2 .. 8; second destinations; a record that holds an error.
Bounds: those of test_splash_gpu.py, and for outputs what rounding P and the result to bf16 gives.
"""
import dataclasses
import math

import numpy as np
import pytest
import torch

import abi_util
from oracle import attention_ref
from tokamax_b200 import _native
from tokamax_b200 import fp8
from tokamax_b200 import splash_attention_kernel as splash
from tokamax_b200 import splash_attention_mask as mask_lib

pytestmark = pytest.mark.gpu

DEV = torch.device("cuda:0")


def _mk(seed, *shape):
  g = torch.Generator().manual_seed(seed)
  return torch.randn(*shape, generator=g).to(torch.bfloat16)


def _dense(mask):
  return np.asarray(mask[(slice(0, mask.shape[0]), slice(0, mask.shape[1]))]).astype(np.bool_)


def _table(sq, skv):
  m = np.random.default_rng(3).random((sq, skv)) < 0.4
  m[:, : skv // 2] &= (np.arange(sq) % 3 != 0)[:, None]  # rows whose keys are all in the second half
  m[5] = False  # and one without any
  return m


def _out_bound(ro, q, k, v, dense, seg, **kw):
  """P and the result are rounded to bf16, 8 significant bits, so each is off by up to 2^-8 of itself: an output
  by 2^-8 (sum p |v| + |o|), and a fiftieth of that for everything held in fp32."""
  spread, _, _ = attention_ref.attention_reference(q, k, v.abs(), dense, seg, **kw)
  return 1.02 * 2.0 ** -8 * (spread + ro.abs()) + 1e-6


CASES = {
    "causal": (lambda sq, skv: mask_lib.CausalMask((sq, skv), skv - sq), {}),
    "window": (lambda sq, skv: mask_lib.LocalMask((sq, skv), (skv // 3, 0), skv - sq), {}),
    "full_sinks": (lambda sq, skv: mask_lib.FullMask((sq, skv)), dict(sinks=True)),
    "segments": (lambda sq, skv: mask_lib.FullMask((sq, skv)), dict(segments=True, sinks=True)),
    "table": (_table, {}),
    "soft_cap": (lambda sq, skv: mask_lib.CausalMask((sq, skv), skv - sq), dict(cap=20.0, sinks=True)),
    "fixed_max": (lambda sq, skv: mask_lib.FullMask((sq, skv)), dict(fixed=6.0, sinks=True)),
}


@pytest.mark.parametrize("sq,skv,hq,hkv", [(128, 4096, 2, 1), (256, 1280, 3, 3), (384, 2944, 4, 2), (1024, 1024, 4, 2)])
@pytest.mark.parametrize("name", sorted(CASES))
def test_forward_and_gradients(name, sq, skv, hq, hkv):
  make, opt = CASES[name]
  mask = make(sq, skv)
  dense = mask if isinstance(mask, np.ndarray) else _dense(mask)
  d = 64 if name == "window" else 128
  # rows of 16 key tiles and more are shared, kv tiles of 16 (q tile, head) steps and more; none with segment ids
  parts = abi_util.row_parts(mask, 1, hq, hkv, sq, skv, d=d, d_v=d)
  assert (parts[0] > 1) == (skv > 2048 and name != "window") and (parts[1] > 1) == (sq == 1024 and name != "window")
  q, k, v, do = _mk(0, 1, hq, sq, d), _mk(1, 1, hkv, skv, d), _mk(2, 1, hkv, skv, d), _mk(3, 1, hq, sq, d)
  # a jump of the row maximum between parts: the keys of the last tiles carry larger logits
  k[:, :, -256:] *= 4
  config = splash.SplashConfig.get_default()
  if "cap" in opt:
    config = dataclasses.replace(config, attn_logits_soft_cap=opt["cap"])
  kernel = splash.make_splash_mha(mask, q_seq_shards=1, save_residuals=True, config=config)
  sinks = torch.linspace(-1.0, 3.0, hq) if opt.get("sinks") else None
  seg = None
  if opt.get("segments"):
    seg = ((torch.arange(sq) * 3 // sq)[None].int(), (torch.arange(skv) * 3 // skv)[None].int())
  scale = 1 / math.sqrt(d)
  qd, kd, vd = (t.to(DEV).requires_grad_(True) for t in (q, k, v))
  out, res = kernel(qd, kd, vd, None if seg is None else splash.SegmentIds(*(s.to(DEV) for s in seg)),
                    None if sinks is None else sinks.to(DEV), logits_scale=scale,
                    max_logit_value=opt.get("fixed"))
  out.backward(do.to(DEV))
  kernel.check_errors()
  ref = [attention_ref.attention_reference(q[0], k[0], v[0], dense, None if seg is None else (seg[0][0], seg[1][0]),
                                           scale=scale, attn_logits_soft_cap=opt.get("cap"), sinks=sinks)]
  ro, rlse, rmax = ref[0]
  live = rlse > -1e30
  bound = _out_bound(ro, q[0], k[0], v[0], dense, None if seg is None else (seg[0][0], seg[1][0]), scale=scale,
                     attn_logits_soft_cap=opt.get("cap"), sinks=sinks)
  assert torch.all(((out[0].float().cpu() - ro).abs() <= bound)[live])
  assert torch.all(out[0].float().cpu()[~live] == 0)
  assert (res["logsumexp"][0].cpu() - rlse)[live].abs().max().item() <= 1e-3
  if "fixed" not in opt:
    assert (res["max_logits"][0].cpu() - rmax)[live].abs().max().item() <= 1e-3 * max(1.0, rmax[live].abs().max().item())
  ro, rlse = torch.where(live[..., None], ro, 0.0), torch.where(live, rlse, float("inf"))
  grads = attention_ref.attention_reference_vjp(do[0], q[0], k[0], v[0], dense,
                                                None if seg is None else (seg[0][0], seg[1][0]), ro, rlse, scale=scale,
                                                attn_logits_soft_cap=opt.get("cap"))
  for got, want in zip((qd.grad, kd.grad, vd.grad), grads):
    assert ((got[0].float().cpu() - want).norm() / want.norm()).item() <= 1e-2


@pytest.mark.parametrize("repeatable", [False, True])
@pytest.mark.parametrize("name", sorted(CASES))
def test_gradients_of_one_kv_head(name, repeatable):
  """Few kv tiles, many steps each (q heads x q tiles): the dkv kernels share the tiles."""
  make, opt = CASES[name]
  sq, skv, hq, d = 1152, 640, 8, 64 if name == "window" else 128
  mask = make(sq, skv)
  dense = mask if isinstance(mask, np.ndarray) else _dense(mask)
  q, k, v, do = _mk(0, 1, hq, sq, d), _mk(1, 1, 1, skv, d), _mk(2, 1, 1, skv, d), _mk(3, 1, hq, sq, d)
  config = splash.SplashConfig.get_default()
  if "cap" in opt:
    config = dataclasses.replace(config, attn_logits_soft_cap=opt["cap"])
  kernel = splash.make_splash_mha(mask, q_seq_shards=1, config=config, repeatable_dq=repeatable)
  seg = None
  if opt.get("segments"):
    seg = ((torch.arange(sq) * 3 // sq)[None].int(), (torch.arange(skv) * 3 // skv)[None].int())
  scale = 1 / math.sqrt(d)
  got = []
  for _ in range(2):
    qd, kd, vd = (t.to(DEV).requires_grad_(True) for t in (q, k, v))
    out = kernel(qd, kd, vd, None if seg is None else splash.SegmentIds(*(s.to(DEV) for s in seg)), logits_scale=scale)
    out.backward(do.to(DEV))
    got.append((qd.grad, kd.grad, vd.grad))
  kernel.check_errors()
  assert torch.equal(got[0][1], got[1][1]) and torch.equal(got[0][2], got[1][2])  # dk, dv: always repeatable
  assert not repeatable or torch.equal(got[0][0], got[1][0])
  pair = None if seg is None else (seg[0][0], seg[1][0])
  ro, rlse, _ = attention_ref.attention_reference(q[0], k[0], v[0], dense, pair, scale=scale,
                                                  attn_logits_soft_cap=opt.get("cap"))
  live = rlse > -1e30
  ro, rlse = torch.where(live[..., None], ro, 0.0), torch.where(live, rlse, float("inf"))
  grads = attention_ref.attention_reference_vjp(do[0], q[0], k[0], v[0], dense, pair, ro, rlse, scale=scale,
                                                attn_logits_soft_cap=opt.get("cap"))
  for g, want in zip(got[0], grads):
    assert ((g[0].float().cpu() - want).norm() / want.norm()).item() <= 1e-2


@pytest.mark.parametrize("p_format,rel", [("e4m3", 3e-2), ("f16", 5e-3)])
@pytest.mark.parametrize("sq,skv", [(128, 4096), (384, 2944)])
def test_e4m3_forward(p_format, rel, sq, skv):
  q, k, v = (fp8.quantize_e4m3(_mk(i, 1, 2, n, 128).to(DEV)) for i, n in ((0, sq), (1, skv), (2, skv)))
  mask = mask_lib.CausalMask((sq, skv), skv - sq)
  kernel = splash.make_splash_mha(mask, q_seq_shards=1)
  scale = 1 / math.sqrt(128)
  out, res = fp8.splash_fwd_fp8(kernel, q, k, v, logits_scale=scale, save_residuals=True, p_format=p_format)
  kernel.check_errors()
  deq = [fp8.dequantize_e4m3(t, torch.float32).cpu()[0] for t in (q, k, v)]
  ro, rlse, _ = attention_ref.attention_reference(*deq, _dense(mask), scale=scale)
  assert ((out[0].float().cpu() - ro).norm() / ro.norm()).item() <= rel
  assert (res["logsumexp"][0].cpu() - rlse).abs().max().item() <= 1e-3


def test_parts_without_a_live_key():
  """Every row is live in one tile only, every tile in some row: most parts of a cluster end with sum 0."""
  sq, skv = 256, 4096
  dense = np.zeros((sq, skv), np.bool_)
  dense[np.arange(sq), (np.arange(sq) * 128 + 17) % skv] = True
  q, k, v = _mk(0, 1, 2, sq, 128), _mk(1, 1, 2, skv, 128), _mk(2, 1, 2, skv, 128)
  kernel = splash.make_splash_mha(dense, q_seq_shards=1, save_residuals=True)
  out, res = kernel(q.to(DEV), k.to(DEV), v.to(DEV), logits_scale=0.1)
  kernel.check_errors()
  ro, rlse, _ = attention_ref.attention_reference(q[0], k[0], v[0], dense, scale=0.1)
  assert (out[0].float().cpu() - ro).abs().max().item() <= 1e-2
  assert (res["logsumexp"][0].cpu() - rlse).abs().max().item() <= 1e-3


INF = float("inf")


def _dead_rows(kind):
  """Masks whose query rows have live keys in no part of a cluster, in one part only, or in all."""
  if kind == "shifted":  # the first half of the rows sees nothing and has no schedule entry at all
    return mask_lib.CausalMask((4096, 2048), -2048)
  m = np.zeros((512, 4096), np.bool_)
  m[0:128, 2048:] = True        # query tile 0 is live in the second half of the keys,
  m[::3] = False                # but for every third row;
  m[200, 128 * 5 + 3] = True    # tile 1 has one live row, in a single key tile (fewer entries than parts);
  m[256:384, :] = True          # tile 3, of a live pair, is dead
  return m


@pytest.mark.parametrize("form", ["bf16", "e4m3", "f16"])
@pytest.mark.parametrize("kind", ["shifted", "table"])
def test_infinite_sinks(kind, form):
  """A sink of -inf is a head without one and +inf takes all the weight: dead rows come out 0, also where
  the part that counts the sink holds no live key.  Their logsumexp is the sink, but for a sink of -inf in
  tiles that hold other rows' keys: there it is the mask value, as for any row without a live key."""
  mask = _dead_rows(kind)
  dense = mask if isinstance(mask, np.ndarray) else _dense(mask)
  sq, skv = dense.shape
  q, k, v = _mk(0, 1, 3, sq, 128), _mk(1, 1, 1, skv, 128), _mk(2, 1, 1, skv, 128)
  sinks = torch.tensor([-INF, INF, 0.5])
  kernel = splash.make_splash_mha(mask, q_seq_shards=1, save_residuals=True)
  if form == "bf16":
    out, res = kernel(q.to(DEV), k.to(DEV), v.to(DEV), None, sinks.to(DEV), logits_scale=0.09)
    rel = 5e-3
  else:
    qkv = [fp8.quantize_e4m3(t.to(DEV)) for t in (q, k, v)]
    out, res = fp8.splash_fwd_fp8(kernel, *qkv, sinks=sinks.to(DEV), logits_scale=0.09, save_residuals=True, p_format=form)
    q, k, v = (fp8.dequantize_e4m3(t, torch.float32).cpu() for t in qkv)
    rel = 3e-2 if form == "e4m3" else 5e-3
  kernel.check_errors()
  out, lse = out[0].float().cpu(), res["logsumexp"][0].cpu()
  live = torch.from_numpy(dense.any(-1))
  assert torch.all(out[:, ~live] == 0) and torch.all(out[1] == 0)
  visited = live.view(-1, 128).any(-1).repeat_interleave(128)
  assert torch.all(lse[0, ~visited] == -INF) and torch.all(lse[1] == INF)
  assert torch.all(lse[0, visited & ~live] == max(kernel.mask_value, -3.0e38))
  assert (lse[2, ~live] - 0.5).abs().max().item() <= 1e-5
  for head, sink in ((0, None), (2, sinks[2:])):
    ro, rlse, _ = attention_ref.attention_reference(q[0, head:head + 1], k[0], v[0], dense, scale=0.09, sinks=sink)
    assert ((out[head] - ro[0])[live].norm() / ro[0][live].norm()).item() <= rel
    assert (lse[head] - rlse[0])[live].abs().max().item() <= 1e-3


def test_listed_tiles_without_a_live_key_change_nothing():
  """One mask as tables cut with blocks of 128 and of 512 tokens (whose partial blocks list tiles that are
  empty) and as a device tensor: the parts of a row hold the same live tiles, so every bit agrees."""
  sq, skv = 512, 4096
  rng = np.random.default_rng(11)
  dense = rng.random((sq, skv)) < 0.5
  dense &= np.kron(rng.random((sq // 128, skv // 128)) < 0.6, np.ones((128, 128))).astype(np.bool_)
  dense[np.arange(sq), np.arange(sq) * 8] = True
  q, k, v, do = _mk(0, 1, 4, sq, 128), _mk(1, 1, 1, skv, 128), _mk(2, 1, 1, skv, 128), _mk(3, 1, 4, sq, 128)
  kw = dict(save_residuals=True, repeatable_dq=True)
  blocks = lambda b: dataclasses.replace(splash.SplashConfig.get_default(), block_q=b, block_kv=b, block_kv_compute=b,
                                         block_q_dkv=b, block_kv_dkv=b, block_kv_dkv_compute=b)
  got = []
  for kernel in (splash.make_splash_mha(dense, q_seq_shards=1, config=blocks(128), **kw),
                 splash.make_splash_mha(dense, q_seq_shards=1, config=blocks(512), **kw),
                 splash.make_dynamic_splash_mha(torch.from_numpy(dense).to(DEV), **kw)):
    qd, kd, vd = (t.to(DEV).requires_grad_(True) for t in (q, k, v))
    out, res = kernel(qd, kd, vd, logits_scale=0.09)
    out.backward(do.to(DEV))
    kernel.check_errors()
    got.append((out, res["logsumexp"], qd.grad, kd.grad, vd.grad))
  for other in got[1:]:
    for a, b in zip(got[0], other):
      assert torch.equal(a, b)


def _heads_for(which, n, mask, sq, skv, group):
  """A number of kv heads for which this GPU's launchers take n parts (forward: which = 0, dkv: 1)."""
  heads = [h for h in range(1, 73) if abi_util.row_parts(mask, 1, group * h, h, sq, skv)[which] == n]
  if not heads:
    pytest.skip(f"no call of this mask is cut in {n} parts on this GPU")
  return heads[0]


@pytest.mark.parametrize("n", range(2, 9))
def test_every_number_of_parts_forward(n):
  """Head dims 80 and 120, a last row pair of one tile, sinks, rows that end inside a part's first or last tile."""
  sq, skv = 384, 4096
  mask = mask_lib.LocalMask((sq, skv), (3000, 0), skv - sq)
  h = _heads_for(0, n, mask, sq, skv, 1)
  q, k, v = _mk(0, 1, h, sq, 80), _mk(1, 1, h, skv, 80), _mk(2, 1, h, skv, 120)
  sinks = torch.linspace(-1.0, 2.0, h)
  kernel = splash.make_splash_mha(mask, q_seq_shards=1, save_residuals=True)
  out, res = kernel(q.to(DEV), k.to(DEV), v.to(DEV), None, sinks.to(DEV), logits_scale=0.1)
  kernel.check_errors()
  dense = _dense(mask)
  ro, rlse, rmax = attention_ref.attention_reference(q[0], k[0], v[0], dense, scale=0.1, sinks=sinks)
  bound = _out_bound(ro, q[0], k[0], v[0], dense, None, scale=0.1, sinks=sinks)
  assert torch.all((out[0].float().cpu() - ro).abs() <= bound)
  assert (res["logsumexp"][0].cpu() - rlse).abs().max().item() <= 1e-3
  assert (res["max_logits"][0].cpu() - rmax).abs().max().item() <= 1e-3


@pytest.mark.parametrize("n", range(2, 9))
@pytest.mark.parametrize("repeatable", [False, True])
def test_every_number_of_parts_backward(n, repeatable):
  """Nine q tiles of three q heads on a kv head: the parts begin at another tile for every head."""
  sq, skv, group = 1152, 384, 3
  mask = mask_lib.FullMask((sq, skv))
  h = _heads_for(1, n, mask, sq, skv, group)
  q, k, v, do = _mk(0, 1, group * h, sq, 80), _mk(1, 1, h, skv, 80), _mk(2, 1, h, skv, 120), _mk(3, 1, group * h, sq, 120)
  kernel = splash.make_splash_mha(mask, q_seq_shards=1, repeatable_dq=repeatable)
  qd, kd, vd = (t.to(DEV).requires_grad_(True) for t in (q, k, v))
  kernel(qd, kd, vd, logits_scale=0.1).backward(do.to(DEV))
  kernel.check_errors()
  wants = attention_ref.fwd_bwd(q, k, v, do, _dense(mask), scale=0.1)[3:]
  for got, want in zip((qd.grad, kd.grad, vd.grad), wants):
    assert ((got.float().cpu() - want).norm() / want.norm()).item() <= 1e-2


def test_chunked_rows():
  s, hq, hkv = 4096, 2, 1
  mask = mask_lib.ChunkedCausalMask((s, s), 2500)  # chunks that end inside a tile; rows of 1 .. 20 key tiles
  assert min(abi_util.row_parts(mask, 1, hq, hkv, s, s)) > 1
  q, k, v, do = _mk(0, 1, hq, s, 128), _mk(1, 1, hkv, s, 128), _mk(2, 1, hkv, s, 128), _mk(3, 1, hq, s, 128)
  kernel = splash.make_splash_mha(mask, q_seq_shards=1)
  qd, kd, vd = (t.to(DEV).requires_grad_(True) for t in (q, k, v))
  out = kernel(qd, kd, vd, logits_scale=0.09)
  out.backward(do.to(DEV))
  kernel.check_errors()
  dense = _dense(mask)
  ro, _, _, *wants = attention_ref.fwd_bwd(q, k, v, do, dense, scale=0.09)
  assert torch.all((out.float().cpu() - ro).abs() <= _out_bound(ro[0], q[0], k[0], v[0], dense, None, scale=0.09))
  for got, want in zip((qd.grad, kd.grad, vd.grad), wants):
    assert ((got.float().cpu() - want).norm() / want.norm()).item() <= 1e-2


def test_second_destinations():
  """Rows of shared tiles arrive in the buffers of the ranks that own them as they do in the local tensor
  (two local buffers stand in for two ranks'), and nothing else is touched."""
  hq, hkv, s, d, world, rank = 4, 2, 4096, 128, 2, 1
  q, k, v, do = (_mk(i, 1, h, s, d).to(DEV) for i, h in enumerate((hq, hkv, hkv, hq)))
  mask = mask_lib.CausalMask((s, s))
  assert min(abi_util.row_parts(mask, 1, hq, hkv, s, s)) > 1
  kernel = splash.make_splash_mha(mask, q_seq_shards=1)
  s_loc = s // world

  def receive(heads):
    bufs = [torch.full((1, heads * world, s_loc, d), 7.0, dtype=torch.bfloat16, device=DEV) for _ in range(world)]
    ptrs = torch.tensor([t.data_ptr() for t in bufs], dtype=torch.int64, device=DEV)
    po = _native.SplashPeerOutput()
    po.ptrs, po.base_bytes, po.rows_per_peer = ptrs.data_ptr(), 0, s_loc
    po.stride_b, po.stride_h, po.stride_s, po.head0 = heads * world * s_loc * d, s_loc * d, d, rank * heads
    return bufs, ptrs, po

  recv = [receive(h) for h in (hq, hq, hkv, hkv)]
  _, _, _, o, lse, _, _ = splash.splash_forward(kernel, q, k, v, None, None, 0.09, None, None, 0, o_peer=recv[0][2])
  grads = splash.splash_backward(kernel, q, k, v, o, lse, do, None, None, 0.09, 0, peers=tuple(r[2] for r in recv[1:]))[:3]
  kernel.check_errors()
  assert torch.equal(o, kernel(q, k, v, logits_scale=0.09))
  for (bufs, _, _), local in zip(recv, (o, *grads)):
    heads = local.shape[1]
    for peer, buf in enumerate(bufs):
      assert torch.equal(buf[:, rank * heads:], local[:, :, peer * s_loc:(peer + 1) * s_loc])
      assert (buf[:, :rank * heads] == 7.0).all()


def test_a_raised_error_record_stops_shared_rows():
  """Every CTA of a cluster that finds an error in the record passes the cluster's barriers and writes nothing."""
  s, hq, hkv = 4096, 4, 2
  mask = mask_lib.CausalMask((s, s))
  assert min(abi_util.row_parts(mask, 1, hq, hkv, s, s)) > 1
  kernel = splash.make_splash_mha(mask, q_seq_shards=1)
  q, k, v, do = (_mk(i, 1, h, s, 128).to(DEV) for i, h in enumerate((hq, hkv, hkv, hq)))
  tables = kernel._tables(DEV, 1)  # pylint: disable=protected-access
  tables.error_record[0] = 1
  for fused in (False, True):
    o, lse, dq, dk, dv = abi_util.fwd_bwd(_native.lib(), kernel, q, k, v, do, 0.09, fused=fused, fill=7.0)
    for name, t in (("o", o), ("lse", lse), ("dk", dk), ("dv", dv)):
      assert (t == 7.0).all(), name
  with pytest.raises(_native.SplashError):
    kernel.check_errors()
  out = kernel(q, k, v, logits_scale=0.09)
  kernel.check_errors()
  assert torch.isfinite(out.float()).all()
