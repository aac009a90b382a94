"""Calls from a thread that has made no CUDA call before: it has no current context, although its device
is right, and the first thing a launch does is a driver call that needs one.  A thread that has a context
of its own keeps it."""
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


_OWN_CONTEXT = """
import ctypes as C
from tokamax_b200 import _native
lib, cuda = _native.lib(), C.CDLL("libcuda.so.1")
ctx, now, mem = C.c_void_p(), C.c_void_p(), C.c_uint64()
assert cuda.cuInit(0) == 0 and cuda.cuCtxCreate_v2(C.byref(ctx), 0, 0) == 0
assert cuda.cuMemAlloc_v2(C.byref(mem), C.c_size_t(4096)) == 0
a = _native.SplashFwdArgs()
n = 65535  # batch rows of as many row pairs: more CTAs than a grid takes, which is found after the tensor maps are made
for t, rows in ((a.q, 256 * n), (a.k, 128), (a.v, 128), (a.o, 256 * n)):
  t.data, t.size[:], t.stride[:] = mem.value, (n, 1, rows, 8), (8 * rows, 8 * rows, 8, 1)
a.sched.row_ptr = a.sched.entries = a.error_record = mem.value
a.sched.n_rows, a.scale = n, 1.0
assert lib.splash_fwd(C.byref(a), None) == -7  # too large: nothing is launched
assert cuda.cuCtxGetCurrent(C.byref(now)) == 0
assert now.value == ctx.value, "the thread's context was replaced"
assert cuda.cuMemFree_v2(mem) == 0 and cuda.cuCtxDestroy_v2(ctx) == 0
print("fine")
"""


def test_a_thread_keeps_its_own_context():
  r = subprocess.run([sys.executable, "-c", _OWN_CONTEXT], cwd=_ROOT, capture_output=True, text=True, timeout=300)
  assert r.returncode == 0 and "fine" in r.stdout, r.stderr[-2000:]
