"""How many CTAs share a schedule row: the launchers' rule, asked on the host with given capacities.

GPU (marked), at sizes whose rows are shared: results of calls on a share of the heads are the whole
call's, bit for bit, and so are o, logsumexp and dq of calls on a share of the query rows.
"""
import ctypes
import math

import numpy as np
import pytest
import torch

from tokamax_b200 import _native
from tokamax_b200 import splash_attention_kernel as splash
from tokamax_b200 import splash_attention_mask as mask_lib
from abi_util import _row_args, row_parts

# clusters of n CTAs that 148 SMs hold at a time: in one piece, in GPCs of 16 and 18 SMs, in pairs of SMs lost to each
CAPACITIES = [
    [0, 148, 74, 49, 37, 29, 24, 21, 18],
    [0, 148, 74, 48, 36, 27, 24, 18, 18],
    [0, 148, 72, 44, 33, 26, 20, 16, 15],
]


@pytest.mark.parametrize("clusters", CAPACITIES)
@pytest.mark.parametrize("batch,hq,hkv,s,shards", [(1, 8, 4, 2048, 2), (1, 8, 4, 2048, 4), (2, 16, 16, 4096, 8),
                                                   (1, 64, 8, 8192, 8), (1, 8, 8, 16384, 8)])
def test_head_shards_are_shared_out_as_the_whole_call(batch, hq, hkv, s, shards, clusters):
  mask = mask_lib.CausalMask((s, s))
  whole = row_parts(mask, batch, hq, hkv, s, s, clusters=clusters)
  assert min(whole) >= 1
  assert row_parts(mask, batch, hq, hkv, s, s, head_shards=shards, clusters=clusters) == whole
  if (hq, s, shards) == (8, 2048, 2):  # a rank's launch by itself would be cut otherwise
    assert row_parts(mask, batch, hq // 2, hkv // 2, s, s, clusters=clusters) != whole and min(whole) > 1


@pytest.mark.parametrize("clusters", CAPACITIES)
@pytest.mark.parametrize("sq,skv,shards", [(2048, 4096, 2), (768, 4096, 2), (1920, 8192, 5), (512, 16384, 4)])
def test_query_shards_are_shared_out_as_the_whole_call(sq, skv, shards, clusters):
  for mask in (mask_lib.CausalMask((sq, skv), skv - sq), mask_lib.LocalMask((sq, skv), (skv // 2, 0), skv - sq),
               mask_lib.FullMask((sq, skv))):
    whole, _ = row_parts(mask, 1, 8, 4, sq, skv, clusters=clusters)
    assert whole > 1 and row_parts(mask, 1, 8, 4, sq, skv, q_shards=shards, clusters=clusters)[0] == whole


@pytest.mark.parametrize("clusters", CAPACITIES)
@pytest.mark.parametrize("batch,hq,hkv,s", [(2, 20, 5, 4096), (1, 20, 5, 8192), (2, 30, 5, 4096), (1, 40, 10, 4096), (1, 32, 8, 4096)])
def test_rows_of_tables_are_not_cut_up_for_waves(batch, hq, hkv, s, clusters):
  """Two or three kv tiles an SM: rows of a table may have every length, which whole tiles, longest first, even out."""
  assert row_parts(mask_lib.FullMask((s, s)), batch, hq, hkv, s, s, clusters=clusters)[1] == 1


# as a B200 reports them
B200 = [0, 148, 74, 45, 33, 26, 22, 15, 15]


@pytest.mark.parametrize("which,window,batch,hq,hkv,sq,skv,best", [
    (0, 0, 1, 2, 1, 3328, 3328, 5), (0, 0, 1, 6, 2, 3072, 3072, 2), (0, 0, 1, 4, 4, 1408, 4096, 5), (0, 0, 1, 8, 8, 1408, 3456, 2),
    (0, 2533, 1, 3, 1, 2816, 2816, 4), (0, 0, 3, 16, 16, 384, 14464, 4), (1, 0, 1, 15, 5, 1152, 1152, 3), (1, 3403, 1, 6, 2, 2304, 2304, 4),
    (1, 0, 4, 12, 2, 640, 640, 3), (1, 0, 1, 16, 2, 1408, 10240, 1), (1, 1368, 3, 16, 2, 4736, 4736, 2)])
def test_grids_a_little_above_what_is_resident(which, window, batch, hq, hkv, sq, skv, best):
  """Calls whose every number of CTAs was measured: the fastest one."""
  mask = mask_lib.LocalMask((sq, skv), (window, 0), skv - sq) if window else mask_lib.CausalMask((sq, skv), skv - sq)
  assert row_parts(mask, batch, hq, hkv, sq, skv, clusters=B200)[which] == best


@pytest.mark.parametrize("batch,hq,hkv,s,parts", [(1, 1, 1, 8192, (7, 4, 4)), (1, 2, 1, 4096, (4, 4, 4)), (1, 2, 1, 16384, (4, 4, 4)),
                                                  (3, 1, 1, 5632, (4, 3, 2)), (1, 8, 8, 4096, (1, 1, 1)), (4, 1, 1, 2432, (3, 3, 3))])
def test_e4m3_rows_are_cut_up_as_they_were(batch, hq, hkv, s, parts):
  """Probabilities of 4 bits: with another number of CTAs a row, results differ by more than the order of fp32 sums."""
  fa, _, shards = _row_args(mask_lib.CausalMask((s, s)), batch, hq, hkv, s, s)
  fa.q.dtype = 2  # SPLASH_F8E4M3
  for clusters, want in zip(CAPACITIES, parts):
    assert _native.lib().splash_fwd_row_parts(ctypes.byref(fa), ctypes.byref(shards), (ctypes.c_int32 * 9)(*clusters)) == want


def test_query_shards_say_whether_their_rows_are_in_order():
  s, cpu = 512, torch.device("cpu")
  kernel = splash.make_splash_mha(mask_lib.CausalMask((s, s)), q_seq_shards=2)
  first, second = (splash._DeviceTables(kernel, cpu, i) for i in range(2))  # pylint: disable=protected-access
  assert first.q_shards == second.q_shards == 2 and first.q_sequence is None
  assert second.q_sequence.tolist() == list(range(s // 2, s))
  mask = mask_lib.CausalMask((s, s))
  mask.q_sequence = np.concatenate([np.arange(256), np.arange(256, 512)[::-1]]).astype(np.int32)
  kernel = splash.make_splash_mha(mask, q_seq_shards=2)
  for i in range(2):  # rows of another order: not shared, in either shard
    tables = splash._DeviceTables(kernel, cpu, i)  # pylint: disable=protected-access
    assert tables.q_shards == 1 and tables.q_sequence.tolist() == mask.q_sequence[256 * i:256 * (i + 1)].tolist()


@pytest.mark.parametrize("chunk,span", [(512, 6), (1000, 10), (4096, 32), (8192, 64), (20000, 64)])
def test_chunked_rows_count_the_keys_they_see(chunk, span):
  """A row of a chunked mask is a chunk long at most; as many steps of a causal mask are shared alike."""
  s = 8192
  got = row_parts(mask_lib.ChunkedCausalMask((s, s), chunk), 1, 2, 2, s, s, clusters=CAPACITIES[1])
  causal = row_parts(mask_lib.CausalMask((s, s)), 1, 2, 2, s, s, clusters=CAPACITIES[1])
  assert got == (1, 1) if span < 16 else min(got) > 1
  if chunk >= s:
    assert got == causal


def test_row_parts_refuses_what_it_cannot_read():
  lib = _native.lib()
  mask = mask_lib.CausalMask((2048, 2048))
  assert lib.splash_fwd_row_parts(None, None, None) == -1 and lib.splash_bwd_row_parts(None, None, None) == -1
  assert lib.splash_fwd_shard(None, None, None) == -1 and lib.splash_bwd_shard(None, None, None) == -1
  assert lib.splash_fwd_fp8_shard(None, None, None) == -1
  assert row_parts(mask, 0, 8, 4, 2048, 2048, clusters=CAPACITIES[0]) == (-1, -1)
  assert row_parts(mask, 1, 8, 4, 2000, 2048, clusters=CAPACITIES[0]) == (-1, -1)
  assert row_parts(mask, 1, 8, 4, 2048, 2048, clusters=[0] * 9) == (-1, -1)
  assert row_parts(mask, 1, 8, 4, 2048, 2048, d=192, clusters=CAPACITIES[0]) == (1, 1)  # the kernels above 128
  kernel = splash.make_splash_mha(mask, q_seq_shards=1)
  assert kernel.head_shards == 1 and kernel.head_shard(4).head_shard(2).head_shards == 8
  for bad in (0, -1, 1 << 16):
    with pytest.raises(ValueError):
      kernel.head_shard(bad)


@pytest.mark.gpu
@pytest.mark.parametrize("repeatable", [True, False])
@pytest.mark.parametrize("name,b,hq,hkv,sq,skv,shards", [("causal", 1, 8, 4, 2048, 2048, 2), ("causal", 1, 8, 4, 2048, 2048, 4),
                                                         ("window", 2, 4, 2, 384, 4096, 2), ("full", 1, 32, 8, 256, 4096, 2)])
def test_shares_of_the_heads_give_the_whole_calls_bits(name, b, hq, hkv, sq, skv, shards, repeatable):
  dev = torch.device("cuda:0")
  mask = {"causal": lambda: mask_lib.CausalMask((sq, skv), skv - sq),
          "window": lambda: mask_lib.LocalMask((sq, skv), (skv * 3 // 4, 0), skv - sq),
          "full": lambda: mask_lib.FullMask((sq, skv))}[name]()
  g = torch.Generator().manual_seed(7)
  mk = lambda h, s: torch.randn(b, h, s, 128, generator=g).to(torch.bfloat16).to(dev)
  q, k, v, do = mk(hq, sq), mk(hkv, skv), mk(hkv, skv), mk(hq, sq)
  kernel = splash.make_splash_mha(mask, q_seq_shards=1, save_residuals=True, repeatable_dq=repeatable)

  def call(kern, *tensors):
    *qkv, d_o = (t.clone() for t in tensors)
    qkv = [t.requires_grad_(True) for t in qkv]
    out, res = kern(*qkv, logits_scale=1 / math.sqrt(128))
    out.backward(d_o)
    return (out, res["logsumexp"], res["max_logits"], *(t.grad for t in qkv))

  whole = call(kernel, q, k, v, do)
  # the case tests what it says only where rows are shared, and a share by itself would not do
  assert max(row_parts(mask, b, hq, hkv, sq, skv)) > 1
  assert row_parts(mask, b, hq, hkv, sq, skv, head_shards=shards) == row_parts(mask, b, hq, hkv, sq, skv)
  assert row_parts(mask, b, hq // shards, hkv // shards, sq, skv) != row_parts(mask, b, hq, hkv, sq, skv)
  for rank in range(shards):
    heads = lambda t: t[:, rank * t.shape[1] // shards:(rank + 1) * t.shape[1] // shards]  # noqa: B023
    share = call(kernel.head_shard(shards), *map(heads, (q, k, v, do)))
    for i, (got, want) in enumerate(zip(share, map(heads, whole))):
      if i == 3 and not repeatable:  # the fused backward's dq: fp32 sums in varying order
        assert ((got.float() - want.float()).norm() / want.float().norm()).item() <= 1e-3
      else:
        assert torch.equal(got, want)
  kernel.check_errors()


@pytest.mark.gpu
@pytest.mark.parametrize("name", ["causal", "window", "full", "table"])
@pytest.mark.parametrize("sq,skv,shards", [(1024, 4096, 4), (768, 2944, 2)])  # 3 q tiles a shard: other pairs than the whole's
def test_shares_of_the_query_rows_give_the_whole_calls_bits(name, sq, skv, shards):
  dev = torch.device("cuda:0")
  table = np.random.default_rng(5).random((sq, skv)) < 0.3
  table[:, 512:1024] = False
  mask = {"causal": lambda: mask_lib.CausalMask((sq, skv), skv - sq),
          "window": lambda: mask_lib.LocalMask((sq, skv), (skv * 3 // 4, 0), skv - sq),
          "full": lambda: mask_lib.FullMask((sq, skv)), "table": lambda: mask_lib.NumpyMask(table)}[name]()
  g = torch.Generator().manual_seed(9)
  mk = lambda h, s: torch.randn(1, h, s, 128, generator=g).to(torch.bfloat16).to(dev)
  q, k, v, do = mk(4, sq), mk(2, skv), mk(2, skv), mk(4, sq)
  kw = dict(save_residuals=True, repeatable_dq=True)
  whole, cut = (splash.make_splash_mha(mask, q_seq_shards=n, **kw) for n in (1, shards))
  assert row_parts(mask, 1, 4, 2, sq, skv)[0] > 1

  def call(kern, rows, **kwargs):
    qi = q[:, :, rows].clone().requires_grad_(True)
    out, res = kern(qi, k, v, logits_scale=0.09, **kwargs)
    out.backward(do[:, :, rows])
    kern.check_errors()
    return out, qi.grad, res["logsumexp"][..., None], res["max_logits"][..., None]

  want = call(whole, slice(0, sq))
  for i in range(shards):
    rows = slice(i * sq // shards, (i + 1) * sq // shards)
    for got, ref in zip(call(cut, rows, q_shard=i), want):
      assert torch.equal(got, ref[:, :, rows])
