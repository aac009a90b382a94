"""What the host side of a call refuses before anything is launched: tensors whose addresses the kernels could not follow."""
import ctypes

import pytest
import torch

from tokamax_b200 import _native
from tokamax_b200 import fp8
from tokamax_b200 import splash_attention_kernel as splash
from tokamax_b200 import splash_attention_mask as mask_lib

S, D = 128, 64


def _bf16(device="cpu", dtype=torch.bfloat16):
  return torch.zeros(1, 1, S, D, dtype=dtype, device=device)


def _ids(device="cpu"):
  return torch.zeros(1, S, dtype=torch.int32, device=device)


def _forward(q=None, k=None, v=None, q_seg=None, kv_seg=None, q_sequence=None, sinks=None, max_logit=None, err=None):
  q, k, v = (_bf16() if t is None else t for t in (q, k, v))
  sched, mask = _native.SplashDeviceSchedule(), _native.SplashMaskFn()
  _native.host().forward(q, k, v, q_seg, kv_seg, q_sequence, sinks, max_logit, torch.zeros(4, dtype=torch.int32) if err is None else err,
                         ctypes.addressof(sched), ctypes.addressof(mask), 1.0, -1e30, 0.0, 1, 1, 0)


def _backward(o=None, lse=None, d_o=None, q_seg=None):
  o, d_o = (_bf16() if t is None else t for t in (o, d_o))
  sched, mask = _native.SplashDeviceSchedule(), _native.SplashMaskFn()
  _native.host().backward(_bf16(), _bf16(), _bf16(), o, torch.zeros(1, 1, S) if lse is None else lse, d_o, q_seg, q_seg, None,
                          torch.zeros(4, dtype=torch.int32), *[ctypes.addressof(sched)] * 2, ctypes.addressof(mask), 1.0, 0.0,
                          True, 1, 1, 0, 0, 0)


@pytest.mark.parametrize("name", ["k", "v", "q_seg", "kv_seg", "q_sequence", "sinks", "max_logit", "err"])
def test_forward_operands_of_another_device_are_refused(name):
  other = _bf16("meta") if name in "kv" else _ids("meta")
  with pytest.raises(RuntimeError, match="on the device of q, cpu, got one on meta"):
    _forward(**{name: other})


@pytest.mark.parametrize("name", ["o", "d_o", "lse", "q_seg"])
def test_backward_operands_of_another_device_are_refused(name):
  other = _bf16("meta") if name in ("o", "d_o") else _ids("meta")
  with pytest.raises(RuntimeError, match="on the device of q, cpu, got one on meta"):
    _backward(**{name: other})


@pytest.mark.parametrize("dtype", [torch.float16, torch.float32, torch.int8])
def test_operands_of_another_type_are_refused(dtype):
  for name in ("q", "k", "v"):
    with pytest.raises(RuntimeError, match="bfloat16"):
      _forward(**{name: _bf16(dtype=dtype)})
  for name in ("o", "d_o"):
    with pytest.raises(RuntimeError, match="bfloat16"):
      _backward(**{name: _bf16(dtype=dtype)})
  kernel = splash.make_splash_mha(mask_lib.CausalMask((S, S)), q_seq_shards=1)
  with pytest.raises(NotImplementedError, match="bfloat16"):
    kernel(_bf16()[0], _bf16()[0], _bf16(dtype=dtype)[0])


def test_e4m3_operands_of_another_device_are_refused():
  kernel = splash.make_splash_mha(mask_lib.CausalMask((S, S)), q_seq_shards=1)
  make = lambda data, scale: fp8.Fp8Tensor(torch.zeros(1, 1, S, 128, device=data).to(torch.float8_e4m3fn), torch.ones(1, 1, 1, device=scale))
  here = make("cpu", "cpu")
  for args in ((here, make("meta", "meta"), here), (here, here, make("cpu", "meta")), (make("cpu", "meta"), here, here)):
    with pytest.raises(ValueError, match="on meta"):
      fp8.splash_fwd_fp8(kernel, *args)
