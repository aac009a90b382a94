"""Calls from a thread that has made no CUDA call before: it has no current context, although its device
is right, and the first thing a launch does is a driver call that needs one."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
_PROGRAM = """
import sys, threading, torch
from tokamax_b200 import splash_attention_kernel as splash
from tokamax_b200 import splash_attention_mask as mask_lib
kernel = splash.make_splash_mha(mask_lib.FullMask((128, 128)), q_seq_shards=1)
q, k, v = (torch.randn(1, 2, 128, 64, device="cuda").to(torch.bfloat16).requires_grad_(True) for _ in range(3))
failed = []
def call():
  try:
    with torch.no_grad():
      kernel(q, k, v)
  except Exception as e:
    failed.append(e)
if sys.argv[1] == "backward":
  do = torch.randn(1, 2, 128, 64, device="cuda").to(torch.bfloat16)
  kernel(q, k, v).backward(do)  # in autograd's thread
  assert torch.isfinite(q.grad.float()).all()
else:
  kernel(q, k, v)
  t = threading.Thread(target=call)
  t.start()
  t.join()
kernel.check_errors()
assert not failed, failed
print("fine")
"""


@pytest.mark.parametrize("what", ["backward", "forward"])
def test_first_cuda_call_of_a_thread(what):
  r = subprocess.run([sys.executable, "-c", _PROGRAM, what], cwd=_ROOT, capture_output=True, text=True, timeout=300)
  assert r.returncode == 0 and "fine" in r.stdout, r.stderr[-2000:]
