"""The host side of a call (csrc/splash_torch.cpp): which tensors are read in place, which are copied, what comes back."""
import ctypes
import math

import pytest
import torch

from tokamax_b200 import _native
from tokamax_b200 import splash_attention_kernel as splash
from tokamax_b200 import splash_attention_mask as mask_lib

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")
B, H, S, D = 2, 2, 256, 64


def _tensors(seed=0):
  g = torch.Generator(device=DEV).manual_seed(seed)
  return [torch.randn(B, H, S, D, generator=g, device=DEV).to(torch.bfloat16) for _ in range(4)]


def _run(q, k, v, do):
  kernel = splash.make_splash_mha(mask_lib.CausalMask((S, S)), q_seq_shards=1, repeatable_dq=True)
  q, k, v = (t.detach().requires_grad_(True) for t in (q, k, v))
  out = kernel(q, k, v, logits_scale=1 / math.sqrt(D))
  grads = torch.autograd.grad(out, (q, k, v), do)
  kernel.check_errors()
  return (out, *grads)


def _like(t, form):
  """The values of ``t`` in another layout."""
  if form == "rows of 68":  # strides that are no multiple of 16 bytes
    wide = torch.zeros(B, H, S, D + 4, dtype=t.dtype, device=DEV)
    view = wide[..., :D]
  elif form == "columns first":  # innermost stride is not 1
    view = torch.zeros(B, H, D, S, dtype=t.dtype, device=DEV).transpose(-1, -2)
  else:  # tokens first: read in place
    view = torch.zeros(B, S, H, D, dtype=t.dtype, device=DEV).transpose(1, 2)
  return view.copy_(t)


@pytest.mark.parametrize("which", range(4))
@pytest.mark.parametrize("form", ["rows of 68", "columns first", "tokens first"])
def test_layouts_give_the_results_of_contiguous_tensors(which, form):
  plain = _tensors()
  other = list(plain)
  other[which] = _like(plain[which], form)
  assert not other[which].is_contiguous()
  for got, want in zip(_run(*other), _run(*plain)):
    assert torch.equal(got, want)


def test_an_expanded_output_gradient():
  q, k, v, _ = _tensors()
  one = torch.ones((), dtype=torch.bfloat16, device=DEV).expand(B, H, S, D)
  for got, want in zip(_run(q, k, v, one), _run(q, k, v, one.contiguous())):
    assert torch.equal(got, want)


def test_other_ranks_are_refused():
  q, k, v, do = _tensors()
  kernel = splash.make_splash_mha(mask_lib.CausalMask((S, S)), q_seq_shards=1)
  for at in range(3):
    bad = [q, k, v]
    bad[at] = bad[at][0]
    with pytest.raises(Exception):  # by the checks of shapes, or by the module's own
      kernel(*bad)
  _, _, _, o, lse, _, _ = splash.splash_forward(kernel, q, k, v, None, None, 0.1, None, None)
  with pytest.raises(RuntimeError, match="rank 4"):
    splash.splash_backward(kernel, q, k, v, o, lse, do[0], None, None, 0.1)
  with pytest.raises(RuntimeError, match="rank 4"):
    splash.splash_forward(kernel, q, k, v[0], None, None, 0.1, None, None)
  kernel.check_errors()


class _Named(torch.Tensor):
  pass


@pytest.mark.parametrize("copied", [False, True])
def test_results_keep_a_tensor_subclass(copied):
  q, k, v, do = _tensors()
  if copied:
    q, k, v = (_like(t, "rows of 68") for t in (q, k, v))
  plain = _run(q, k, v, do)
  named = _run(*(t.as_subclass(_Named) for t in (q, k, v)), do)
  assert [type(t) for t in named] == [_Named] * 4
  for got, want in zip(named, plain):
    assert torch.equal(got.as_subclass(torch.Tensor), want)
  params = _run(*(torch.nn.Parameter(t) for t in (q, k, v)), do)
  assert all(type(t) is torch.Tensor for t in params)


def test_operands_of_another_device_are_refused():
  q, k, v, _ = _tensors()
  kernel = splash.make_splash_mha(mask_lib.CausalMask((S, S)), q_seq_shards=1)
  want = kernel(q, k, v, logits_scale=0.125)
  for args in ((q, k.cpu(), v), (q, k, v.cpu())):
    with pytest.raises(RuntimeError, match="on the device of q"):
      kernel(*args, logits_scale=0.125)
  assert torch.equal(kernel(q, k, v, logits_scale=0.125), want)


# ---- the autograd function in native code, against the python one, which calls with a fixed maximum and others still take
def _both(monkeypatch, run):
  native = run()
  with monkeypatch.context() as m:
    m.setattr(splash, "_plain", lambda *_: False)
    m.setattr(splash, "_in_class_of", lambda source, result: result)
    python = run()
  return native, python


@pytest.mark.parametrize("d", [64, 256])
@pytest.mark.parametrize("soft_cap,repeatable", [(None, True), (20.0, True)])
@pytest.mark.parametrize("wanted", [(0, 1, 2), (0,), (1,), (2,)])
def test_native_and_python_autograd_functions_agree(monkeypatch, d, soft_cap, repeatable, wanted):
  g = torch.Generator(device=DEV).manual_seed(d)
  q, k, v, do = (torch.randn(B, h, S, d, generator=g, device=DEV).to(torch.bfloat16) for h in (4, 2, 2, 4))
  config = splash.dataclasses.replace(splash.SplashConfig.get_default(), attn_logits_soft_cap=soft_cap)
  kernel = splash.make_splash_mha(mask_lib.CausalMask((S, S)), config=config, q_seq_shards=1, repeatable_dq=repeatable,
                                  save_residuals=True)

  def run():
    ts = [t.detach().requires_grad_(i in wanted) for i, t in enumerate((q, k, v))]
    out, res = kernel(*ts, logits_scale=d ** -0.5)
    assert out.requires_grad and not res["logsumexp"].requires_grad and not res["max_logits"].requires_grad
    return (out, res["logsumexp"], res["max_logits"], *torch.autograd.grad(out, [ts[i] for i in wanted], do))

  for got, want in zip(*_both(monkeypatch, run)):
    assert torch.equal(got, want)
  for mode in (torch.no_grad, torch.inference_mode):
    with mode():
      out, res = kernel(q, k, v, logits_scale=d ** -0.5)
    assert not out.requires_grad and torch.equal(out, run()[0])


def test_the_native_function_saves_its_tensors_through_hooks(monkeypatch):
  q, k, v, do = _tensors()
  kernel = splash.make_splash_mha(mask_lib.CausalMask((S, S)), q_seq_shards=1, repeatable_dq=True)

  def run():
    ts = [t.detach().requires_grad_(True) for t in (q, k, v)]
    packed = []
    pack = lambda t: (packed.append(t.shape), t.cpu())[1]
    with torch.autograd.graph.saved_tensors_hooks(pack, lambda t: t.to(DEV)):
      out = kernel(*ts, logits_scale=0.125)
    first = torch.autograd.grad(out, ts, do, retain_graph=True)
    second = torch.autograd.grad(out, ts, do)
    with pytest.raises(RuntimeError, match="a second time"):
      torch.autograd.grad(out, ts, do)
    assert packed == [q.shape, k.shape, v.shape, out.shape, out.shape[:3]]
    assert all(torch.equal(a, b) for a, b in zip(first, second))
    return first

  for got, want in zip(*_both(monkeypatch, run)):
    assert torch.equal(got, want)


def test_a_saved_operand_that_was_written_to_is_refused():
  q, k, v, do = _tensors()
  kernel = splash.make_splash_mha(mask_lib.CausalMask((S, S)), q_seq_shards=1)
  ts = [t.detach().requires_grad_(True) for t in (q, k, v)]
  out = kernel(*ts, logits_scale=0.125)
  with torch.no_grad():
    ts[1].zero_()
  with pytest.raises(RuntimeError, match="modified by an inplace operation"):
    torch.autograd.grad(out, ts, do)


def test_transforms_are_refused_as_before():
  q, k, v, _ = _tensors()
  kernel = splash.make_splash_mha(mask_lib.CausalMask((S, S)), q_seq_shards=1)
  call = lambda *t: kernel(*t, logits_scale=0.125)
  with pytest.raises(RuntimeError):
    torch.func.vmap(lambda x: call(x, k, v))(q[None])
  with pytest.raises(RuntimeError):
    torch.func.grad(lambda x: call(x, k, v).float().sum())(q)
  with torch.autograd.forward_ad.dual_level(), pytest.raises((RuntimeError, NotImplementedError)):
    call(torch.autograd.forward_ad.make_dual(q, torch.ones_like(q)), k, v)


def test_statuses_arrive_as_the_packages_exception():
  q, k, v, do = _tensors()
  kernel = splash.make_splash_mha(mask_lib.CausalMask((S, S)), q_seq_shards=1)
  ts = [t.detach().requires_grad_(True) for t in (q, k, v)]
  with pytest.raises(_native.SplashError, match="splash_fwd") as info:  # a scale of zero
    kernel(*ts, logits_scale=0.0)
  assert info.value.status == -1
  out = kernel(*ts, logits_scale=0.125)
  lib, address = _native.lib(), lambda f: ctypes.cast(f, ctypes.c_void_p).value
  refuse = ctypes.CFUNCTYPE(ctypes.c_int, ctypes.c_void_p, ctypes.c_void_p, ctypes.c_void_p)(lambda *_: -2)
  rest = (lib.splash_bwd_workspace_bytes, lib.splash_bwd_fused_workspace_bytes)
  bind = lambda bwd: _native.host().bind_library(*(address(f) for f in (lib.splash_fwd_shard, bwd, *rest)))
  bind(refuse)
  try:
    with pytest.raises(_native.SplashError, match="splash_bwd") as info:
      torch.autograd.grad(out, ts, do)
    assert info.value.status == -2
  finally:
    bind(lib.splash_bwd_shard)
  assert all(g.isfinite().all() for g in torch.autograd.grad(kernel(*ts, logits_scale=0.125), ts, do))
