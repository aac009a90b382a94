"""The host side of a call (csrc/splash_torch.cpp): which tensors are read in place, which are copied, what comes back."""
import math

import pytest
import torch

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
