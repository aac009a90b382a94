"""Timing cases of splash attention: what programs ask of the public entry points, and in which sizes.

A case is a dict of plain values.  ``kind`` says which entry point it goes through:

  prefill  kernel object, forward only, ``[B, H, S, D]`` bf16 (inference; a kv cache longer than the
           q rows for chunked prefill)
  train    kernel object, forward and the gradients of q, k and v
  fp8      block-scaled e4m3 forward (inference prefill from a quantised cache)
  op       ``dot_product_attention`` on ``[B, T, N, H]`` tensors, forward and gradients

``mask`` is ``causal`` (the last q row sees the last key), ``local`` (causal with a window to the
left), ``full``, or ``prefix`` (a bool tensor on the device: a bidirectional prefix, causal behind
it).  ``docs`` > 0 packs documents of docs / 8 .. docs tokens into each row (segment ids).
"""

import math
import random

import numpy as np
import torch

from tokamax_b200 import fp8
from tokamax_b200 import op
from tokamax_b200 import splash_attention_kernel as splash
from tokamax_b200 import splash_attention_mask as mask_lib

_DEFAULTS = dict(kind="train", mask="causal", batch=1, q_len=1024, kv_len=0, q_heads=8, kv_heads=8, d=128, d_v=0,
                 window=0, docs=0, soft_cap=0.0, sinks=False, repeatable=False, p_format="")


def _case(**kw):
  c = dict(_DEFAULTS, **kw)
  c["kv_len"] = c["kv_len"] or c["q_len"]
  c["d_v"] = c["d_v"] or c["d"]
  return c


def listed():
  return [
      # The first tokens of a chat turn in a small model: a handful of CTAs, all latency and launches.
      _case(name="prefill_short", kind="prefill", q_len=256, q_heads=8, kv_heads=2, d=64),
      # A chunk of a long prompt against the cache that earlier chunks filled: few q rows, many keys.
      _case(name="prefill_chunk", kind="prefill", q_len=512, kv_len=16384, q_heads=32, kv_heads=8),
      # Serving with attention sinks and a sliding window, head dim 64, an odd number of q tiles.
      _case(name="prefill_window_sinks", kind="prefill", mask="local", window=1024, batch=2, q_len=6016, q_heads=64,
            kv_heads=8, d=64, sinks=True),
      # The parity-size training step (small models, fine-tuning on short rows).
      _case(name="train_short", batch=2, q_len=1024, q_heads=8, kv_heads=8),
      # Pretraining at 8K context with grouped heads: the benchmark's default workload, and the largest step.
      _case(name="train_gqa_8k", batch=4, q_len=8192, q_heads=32, kv_heads=8),
      # Packed-sequence pretraining: sliding window and documents cut from a packed row.
      _case(name="train_packed_window", mask="local", window=4096, docs=4096, batch=8, q_len=16384, q_heads=16,
            kv_heads=16),
      # Bitwise repeatable gradients, one kv head per row (MQA), head dim 64.
      _case(name="train_repeatable_mqa", batch=2, q_len=4096, q_heads=16, kv_heads=1, d=64, repeatable=True),
      # The two head-dim pairs above 128 that the repository's tests and benchmark carry.
      _case(name="train_hd256", q_len=8192, q_heads=16, kv_heads=8, d=256),
      _case(name="train_hd192_128", q_len=4096, q_heads=32, kv_heads=32, d=192, d_v=128),
      # Long-prompt prefill from an e4m3 cache.
      _case(name="fp8_prefill_32k", kind="fp8", batch=2, q_len=32768, q_heads=32, kv_heads=8, p_format="e4m3"),
      # Op layout with everything odd at once: 13 q tiles, a head dim of 80, 12 heads, soft cap, a window.
      _case(name="op_softcap_ragged", kind="op", mask="local", window=768, batch=3, q_len=1664, q_heads=12, kv_heads=4,
            d=80, soft_cap=50.0),
      # A mask that is data on the device (prefix language model): schedules are built in the call.
      _case(name="op_prefix_mask", kind="op", mask="prefix", batch=2, q_len=4096, q_heads=16, kv_heads=4),
  ]


# ----------------------------------------------------------------------------------------------
# drawing more cases of the same ranges
# ----------------------------------------------------------------------------------------------
def _len(rng, lo, hi):
  """A multiple of 128 between lo and hi, even over the logarithm."""
  return max(1, round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / 128)) * 128


def _heads(rng, most=32):
  kv = rng.choice([h for h in (1, 2, 3, 4, 5, 8, 12, 16, 32) if h <= most])
  group = rng.choice([g for g in (1, 2, 3, 4, 6, 8) if kv * g <= most])
  return dict(q_heads=kv * group, kv_heads=kv)


def draw(rng: random.Random):
  largest = {}
  for c in listed():
    key = "wide" if c["d"] > 128 else c["kind"]
    largest[key] = max(largest.get(key, 0.0), work(c)["flops"])
  while True:
    family = rng.choice(["prefill", "chunk", "train", "train", "packed", "repeatable", "wide", "fp8", "op", "op_prefix"])
    batch = rng.choice([1, 1, 2, 3, 4, 8])
    window = lambda s: 0 if rng.random() < 0.5 else rng.randrange(100, max(101, s))  # noqa: E731
    if family == "prefill":
      s = _len(rng, 128, 16384)
      w = window(s)
      c = _case(kind="prefill", mask="local" if w else "causal", window=w, batch=batch, q_len=s, d=rng.choice([64, 96, 128]),
                sinks=rng.random() < 0.3, **_heads(rng, 64))
    elif family == "chunk":
      q = _len(rng, 128, 2048)
      c = _case(kind="prefill", batch=batch, q_len=q, kv_len=max(q, _len(rng, 1024, 32768)), d=rng.choice([64, 128, 128]),
                **_heads(rng))
    elif family == "train":
      s = _len(rng, 256, 8192)
      w = window(s)
      c = _case(mask=rng.choice(["causal", "full"]) if not w else "local", window=w, batch=batch, q_len=s,
                d=rng.choice([64, 80, 96, 120, 128, 128, 128]), sinks=rng.random() < 0.2, **_heads(rng))
    elif family == "packed":
      s = _len(rng, 2048, 16384)
      c = _case(mask="local", window=s // rng.choice([2, 4, 8]), docs=s // rng.choice([2, 4, 8]), batch=batch, q_len=s,
                d=rng.choice([64, 128, 128]), **_heads(rng))
    elif family == "repeatable":
      c = _case(batch=batch, q_len=_len(rng, 512, 8192), d=rng.choice([64, 128]), repeatable=True, **_heads(rng))
    elif family == "wide":
      d, d_v = rng.choice([(192, 128), (256, 256), (160, 160)])
      c = _case(batch=batch, q_len=_len(rng, 512, 8192), d=d, d_v=d_v, **_heads(rng))
    elif family == "fp8":
      c = _case(kind="fp8", batch=batch, q_len=_len(rng, 1024, 32768), p_format=rng.choice(["e4m3", "f16"]), **_heads(rng))
    elif family == "op":
      s = _len(rng, 256, 8192)
      w = window(s)
      c = _case(kind="op", mask="local" if w else "causal", window=w, batch=batch, q_len=s, d=rng.choice([64, 72, 80, 112, 128]),
                soft_cap=rng.choice([0.0, 30.0, 50.0]), **_heads(rng))
    else:
      c = _case(kind="op", mask="prefix", batch=batch, q_len=_len(rng, 512, 4096), d=rng.choice([64, 128]), **_heads(rng))
    if work(c)["flops"] <= largest["wide" if c["d"] > 128 else c["kind"]]:
      return c


# ----------------------------------------------------------------------------------------------
# inputs
# ----------------------------------------------------------------------------------------------
def _mask(c):
  shape = (c["q_len"], c["kv_len"])
  offset = c["kv_len"] - c["q_len"]
  if c["mask"] == "causal":
    return mask_lib.CausalMask(shape, offset)
  if c["mask"] == "local":
    return mask_lib.LocalMask(shape, (c["window"], 0), offset)
  return mask_lib.FullMask(shape)


def _segments(c, seed):
  """Documents of docs / 8 .. docs tokens packed into every row, the last one cut off."""
  rng = np.random.default_rng(seed)
  ids = np.zeros((c["batch"], c["q_len"]), np.int32)
  for row in ids:
    at, doc = 0, 0
    while at < row.size:
      n = int(rng.integers(c["docs"] // 8, c["docs"] + 1))
      row[at:at + n] = doc
      at, doc = at + n, doc + 1
  return ids


def prepare(case, seed):
  """What the program holds before the call: inputs on the device, and the kernel object of its mask."""
  c = dict(case)
  dev = torch.device("cuda")
  gen = torch.Generator(device=dev).manual_seed(seed)

  def normal(heads, length, cols):
    shape = (c["batch"], length, heads, cols) if c["kind"] == "op" else (c["batch"], heads, length, cols)
    return torch.randn(shape, generator=gen, device=dev, dtype=torch.float32).to(torch.bfloat16)

  s = {"case": c}
  q, k, v = (normal(c["q_heads"], c["q_len"], c["d"]), normal(c["kv_heads"], c["kv_len"], c["d"]),
             normal(c["kv_heads"], c["kv_len"], c["d_v"]))
  if c["kind"] in ("train", "op"):
    q, k, v = (t.requires_grad_(True) for t in (q, k, v))
    s["do"] = normal(c["q_heads"], c["q_len"], c["d_v"])
  if c["kind"] == "fp8":
    q, k, v = (fp8.quantize_e4m3(t) for t in (q, k, v))
  s.update(q=q, k=k, v=v, scale=c["d"] ** -0.5)
  if c["mask"] == "prefix":
    n = c["q_len"]
    prefix = random.Random(seed).randrange(n // 8, n // 2)
    at = torch.arange(n, device=dev)
    s["mask"] = (at[None, :] <= at[:, None]) | (at[None, :] < prefix)
  elif c["kind"] != "op":
    s["kernel"] = splash.make_splash_mha(_mask(c), q_seq_shards=1, repeatable_dq=c["repeatable"])
  if c["sinks"]:
    s["sinks"] = torch.randn(c["q_heads"], generator=gen, device=dev)
  if c["docs"]:
    ids = torch.from_numpy(_segments(c, seed)).to(dev)
    s["segments"] = splash.SegmentIds(q=ids, kv=ids)
  return s


def run(state):
  """One forward, or one forward and backward, as a program calls it; returns the output and the gradients."""
  c, q, k, v = state["case"], state["q"], state["k"], state["v"]
  if c["kind"] == "prefill":
    with torch.no_grad():
      return state["kernel"](q, k, v, state.get("segments"), state.get("sinks"), logits_scale=state["scale"])
  if c["kind"] == "fp8":
    return fp8.splash_fwd_fp8(state["kernel"], q, k, v, logits_scale=state["scale"], p_format=c["p_format"])
  if c["kind"] == "op":
    if c["mask"] == "prefix":
      out = op.dot_product_attention(q, k, v, mask=state["mask"])
    else:
      out = op.dot_product_attention(q, k, v, is_causal=True, local_window_size=(c["window"], 0) if c["window"] else None,
                                     logits_soft_cap=c["soft_cap"] or None)
  else:
    out = state["kernel"](q, k, v, state.get("segments"), state.get("sinks"), logits_scale=state["scale"])
  dq, dk, dv = torch.autograd.grad(out, (q, k, v), state["do"])
  return {"out": out, "dq": dq, "dk": dk, "dv": dv}


# ----------------------------------------------------------------------------------------------
# what a pass cannot do without, and how exact it is
# ----------------------------------------------------------------------------------------------
def _live_pairs(c):
  """Unmasked (query, key) pairs of all batch rows, per q head (documents and prefixes: of seed 0)."""
  n, m = c["q_len"], c["kv_len"]
  rows = np.arange(n, dtype=np.int64) + (m - n)
  if c["docs"]:
    total = 0
    for ids in _segments(c, 0):
      first = np.searchsorted(ids, ids)  # first token of each token's document
      total += int((rows - np.maximum(first, rows - c["window"]) + 1).sum())
    return total
  if c["mask"] == "full":
    per_row = n * m
  elif c["mask"] == "prefix":
    prefix = random.Random(0).randrange(n // 8, n // 2)
    per_row = int(np.maximum(rows + 1, prefix).sum())
  else:
    left = np.maximum(rows - c["window"], 0) if c["mask"] == "local" else 0
    per_row = int((rows + 1 - left).sum())
  return c["batch"] * per_row


def work(case):
  """Mask-counted operations (forward: q k^T and p v; backward: five matmuls) and each input and output once."""
  c = case
  pairs = _live_pairs(c) * c["q_heads"]
  d, d_v = c["d"], c["d_v"]
  grads = c["kind"] in ("train", "op")
  flops = 2.0 * pairs * (d + d_v) + (2.0 * pairs * (3 * d + 2 * d_v) if grads else 0.0)
  size = 1 if c["kind"] == "fp8" else 2
  q_rows, kv_rows = c["batch"] * c["q_heads"] * c["q_len"], c["batch"] * c["kv_heads"] * c["kv_len"]
  inputs = size * (q_rows * d + kv_rows * (d + d_v))
  out = 2 * q_rows * d_v
  nbytes = inputs + out + (inputs + out if grads else 0)  # dO comes in, dq / dk / dv go out
  if c["mask"] == "prefix":
    nbytes += c["q_len"] * c["kv_len"]
  if c["docs"]:
    nbytes += 4 * c["batch"] * c["q_len"]
  return {"bytes": float(nbytes), "flops": flops}


def tolerance(case):
  """bf16: P, dS and every result are rounded to 8 bits; outputs and gradients are 2.3e-3 .. 2.7e-3 (relative
  L2) from the fp32 oracle, and four times that is stated.  e4m3 P: the probabilities themselves have 4 bits
  (the contract of the repository's own tests: 3e-2)."""
  if case["kind"] == "fp8" and case["p_format"] == "e4m3":
    return {"rel": 3e-2, "max": 0.6}
  return {"rel": 1e-2, "max": 0.2}


# ----------------------------------------------------------------------------------------------
# the same results in 64 bits
# ----------------------------------------------------------------------------------------------
_EXACT_ELEMENTS = 1 << 27  # scores held at a time: 1 GiB each of logits, probabilities and their gradients


def _wide(t, c):
  """One operand in 64 bits as [B, H, S, D]; e4m3 values times the scale of their 128-token tile."""
  if isinstance(t, fp8.Fp8Tensor):
    return t.data.double() * t.scale.double().repeat_interleave(fp8.SCALE_TILE, dim=2)[..., None]
  t = t.detach().double()
  return t.transpose(1, 2) if c["kind"] == "op" else t


def _keep(c, state, b, rows, lo, hi):
  """Which keys lo .. hi the query rows of batch row b see: bool [rows, hi - lo]."""
  q_at = (rows + (c["kv_len"] - c["q_len"]))[:, None]
  k_at = torch.arange(lo, hi, device=rows.device)[None, :]
  if c["mask"] == "prefix":
    return state["mask"][rows, lo:hi]
  if c["mask"] == "full":
    return torch.ones((rows.numel(), hi - lo), dtype=torch.bool, device=rows.device)
  keep = k_at <= q_at
  if c["mask"] == "local":
    keep &= k_at >= q_at - c["window"]
  if c["docs"]:
    ids = state["segments"].q[b]
    keep &= ids[rows][:, None] == ids[lo:hi][None, :]
  return keep


def exact(case, seed):
  """What ``run`` returns for these inputs, from dense attention in 64 bits, a block of query rows at a time."""
  c = dict(case)
  state = prepare(c, seed)
  q, k, v = (_wide(state[n], c) for n in ("q", "k", "v"))
  grads = c["kind"] in ("train", "op")
  offset, group, dev = c["kv_len"] - c["q_len"], c["q_heads"] // c["kv_heads"], q.device
  out = torch.zeros((c["batch"], c["q_heads"], c["q_len"], c["d_v"]), dtype=torch.float64, device=dev)
  if grads:
    do = _wide(state["do"], c)
    dq, dk, dv = torch.zeros_like(q), torch.zeros_like(k), torch.zeros_like(v)
  for b in range(c["batch"]):
    first = 0
    while first < c["q_len"]:
      n = min(c["q_len"] - first, max(128, _EXACT_ELEMENTS // (c["q_heads"] * c["kv_len"])))
      rows = torch.arange(first, first + n, device=dev)
      lo = max(0, first + offset - c["window"]) if c["mask"] == "local" else 0
      hi = c["kv_len"] if c["mask"] in ("full", "prefix") else first + n + offset
      # heads as [kv heads, group * rows]: the q heads of one kv head are rows of one product
      qb = q[b, :, first:first + n].reshape(c["kv_heads"], group * n, c["d"])
      kb, vb = k[b, :, lo:hi], v[b, :, lo:hi]
      keep = _keep(c, state, b, rows, lo, hi)
      x = (qb @ kb.transpose(1, 2)).mul_(state["scale"]).view(c["kv_heads"], group, n, hi - lo)
      slope = None
      if c["soft_cap"]:
        x.div_(c["soft_cap"]).tanh_()
        slope = 1 - x * x if grads else None
        x.mul_(c["soft_cap"])
      x.masked_fill_(~keep, -math.inf)
      top = x.amax(-1, keepdim=True)
      sink = state["sinks"].double().view(c["kv_heads"], group, 1, 1) if c["sinks"] else None
      if sink is not None:
        top = torch.maximum(top, sink)
      x.sub_(top).exp_()
      total = x.sum(-1, keepdim=True)
      if sink is not None:
        total = total + torch.exp(sink - top)
      p = x.div_(total).view(c["kv_heads"], group * n, hi - lo)
      ob = p @ vb
      out[b, :, first:first + n] = ob.view(c["q_heads"], n, c["d_v"])
      if grads:
        dob = do[b, :, first:first + n].reshape(c["kv_heads"], group * n, c["d_v"])
        dv[b, :, lo:hi] += p.transpose(1, 2) @ dob
        ds = (dob @ vb.transpose(1, 2)).sub_((ob * dob).sum(-1, keepdim=True)).mul_(p).mul_(state["scale"])
        if slope is not None:
          ds.mul_(slope.view_as(ds))
        dq[b, :, first:first + n] = (ds @ kb).view(c["q_heads"], n, c["d"])
        dk[b, :, lo:hi] += ds.transpose(1, 2) @ qb
      first += n
  lay = (lambda t: t.transpose(1, 2).contiguous()) if c["kind"] == "op" else (lambda t: t)
  if not grads:
    return lay(out)
  return {"out": lay(out), "dq": lay(dq), "dk": lay(dk), "dv": lay(dv)}
