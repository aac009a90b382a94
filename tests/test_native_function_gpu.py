"""The autograd function in native code (csrc/splash_torch.cpp): the form of its backward, and calls that are traced, recomputed or
made on a stream of their own."""
import ctypes
import dataclasses

import pytest
import torch
from torch.utils import checkpoint

from tokamax_b200 import _native
from tokamax_b200 import splash_attention_kernel as splash
from tokamax_b200 import splash_attention_mask as mask_lib

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")
B, S = 2, 384


def _operands(d, seed=0):
  g = torch.Generator(device=DEV).manual_seed(seed)
  return [torch.randn(B, h, S, d, generator=g, device=DEV).to(torch.bfloat16) for h in (4, 2, 2, 4)]


def _kernel(soft_cap=None, repeatable=True):
  config = dataclasses.replace(splash.SplashConfig.get_default(), attn_logits_soft_cap=soft_cap)
  return splash.make_splash_mha(mask_lib.CausalMask((S, S)), config=config, q_seq_shards=1, repeatable_dq=repeatable)


def _leaves(*tensors):
  return [t.detach().clone().requires_grad_(True) for t in tensors]


@pytest.fixture
def native_calls(monkeypatch):
  """How often a call went through the native function."""
  calls = []
  own = splash.SplashAttentionKernel._attention  # pylint: disable=protected-access
  monkeypatch.setattr(splash.SplashAttentionKernel, "_attention", lambda *args: (calls.append(1), own(*args))[1])
  return calls


@pytest.fixture
def backward_flags():
  """The flags of every backward launched."""
  lib, flags = _native.lib(), []
  address = lambda f: ctypes.cast(f, ctypes.c_void_p).value
  rest = [address(f) for f in (lib.splash_bwd_workspace_bytes, lib.splash_bwd_fused_workspace_bytes)]

  @ctypes.CFUNCTYPE(ctypes.c_int, ctypes.c_void_p, ctypes.c_void_p, ctypes.c_void_p)
  def record(args, shards, stream):
    flags.append(_native.SplashBwdArgs.from_address(args).flags)
    shards = None if shards is None else ctypes.byref(_native.SplashShards.from_address(shards))
    return lib.splash_bwd_shard(ctypes.byref(_native.SplashBwdArgs.from_address(args)), shards, stream)

  _native.host().bind_library(address(lib.splash_fwd_shard), address(record), *rest)
  yield flags
  _native.host().bind_library(address(lib.splash_fwd_shard), address(lib.splash_bwd_shard), *rest)


@pytest.mark.parametrize("soft_cap", [None, 20.0])
@pytest.mark.parametrize("d,repeatable,fused", [(64, False, True), (80, False, True), (128, False, True), (192, False, False),
                                                (256, False, False), (64, True, False), (128, True, False)])
def test_both_functions_take_the_same_backward(monkeypatch, native_calls, backward_flags, d, repeatable, fused, soft_cap):
  q, k, v, do = _operands(d)
  kernel = _kernel(soft_cap, repeatable)

  def run():
    ts = _leaves(q, k, v)
    return torch.autograd.grad(kernel(*ts, logits_scale=d ** -0.5), ts, do)

  native = run()
  assert len(native_calls) == 1
  with monkeypatch.context() as m:
    m.setattr(splash, "_plain", lambda *_: False)
    m.setattr(splash, "_in_class_of", lambda source, result: result)
    python = run()
  assert len(native_calls) == 1
  assert backward_flags == [_native.BWD_FUSED_DQ if fused else 0] * 2
  for i, (got, want) in enumerate(zip(native, python)):
    if i == 0 and fused:  # fp32 sums in varying order
      assert ((got.float() - want.float()).norm() / want.float().norm()).item() <= 1e-3
    else:
      assert torch.equal(got, want)


def test_on_a_stream_of_its_own():
  q, k, v, do = _operands(64)
  kernel = _kernel()
  call = lambda ts: kernel(*ts, logits_scale=0.125)
  ts = _leaves(q, k, v)
  out = call(ts)
  want = (out, *torch.autograd.grad(out, ts, do))
  stream = torch.cuda.Stream(DEV)
  for _ in range(4):
    ts = _leaves(q, k, v)
    stream.wait_stream(torch.cuda.current_stream(DEV))
    with torch.cuda.stream(stream):
      out = call(ts)
    grads = torch.autograd.grad(out, ts, do)  # the backward follows the forward's stream
    torch.cuda.current_stream(DEV).wait_stream(stream)
    assert all(torch.equal(a, b) for a, b in zip((out, *grads), want))
  kernel.check_errors()


@pytest.mark.parametrize("reentrant", [False, True])
def test_recomputed_by_a_checkpoint(native_calls, reentrant):
  q, k, v, do = _operands(64)
  kernel = _kernel()

  def block(*ts):
    return kernel(*(t * 1.5 for t in ts), logits_scale=0.125) + 1.0

  ts = _leaves(q, k, v)
  out = block(*ts)
  want = (out, *torch.autograd.grad(out, ts, do))
  ts = _leaves(q, k, v)
  out = checkpoint.checkpoint(block, *ts, use_reentrant=reentrant)
  out.backward(do)
  assert len(native_calls) == 3
  assert all(torch.equal(a, b) for a, b in zip((out, *(t.grad for t in ts)), want))
  out = kernel(*ts, logits_scale=0.125)  # (no exception of the recomputation is left over)
  kernel.check_errors()


def test_a_hook_that_raises_is_heard():
  q, k, v, _ = _operands(64)
  kernel = _kernel()

  def pack(_):
    raise KeyError("pack")

  with torch.autograd.graph.saved_tensors_hooks(pack, lambda t: t), pytest.raises(KeyError, match="pack"):
    kernel(*_leaves(q, k, v), logits_scale=0.125)
  assert kernel(*_leaves(q, k, v), logits_scale=0.125).requires_grad


def test_traced_calls_are_recorded(native_calls):
  q, k, v, _ = _operands(64)
  kernel = _kernel()
  call = lambda *ts: kernel(*ts, logits_scale=0.125)
  traced = torch.jit.trace(call, (q, k, v), check_trace=False)
  assert not native_calls
  other = _operands(64, seed=1)[:3]
  assert torch.equal(traced(*other), call(*other))


def test_compiled_calls_give_the_same(native_calls):
  q, k, v, do = _operands(64)
  kernel = _kernel()
  call = lambda *ts: kernel(*ts, logits_scale=0.125) * 2.0
  ts = _leaves(q, k, v)
  out = call(*ts)
  want = (out, *torch.autograd.grad(out, ts, do))
  ts = _leaves(q, k, v)
  out = torch.compile(call, backend="eager")(*ts)
  assert all(torch.equal(a, b) for a, b in zip((out, *torch.autograd.grad(out, ts, do)), want))
