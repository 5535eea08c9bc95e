"""What the decode steps' projections do with their sums (csrc/gemm_rows.cuh): rotated queries, appended keys and values."""

import ctypes

import pytest
import torch

from maxtext_indextts2_b200 import _lib

pytestmark = pytest.mark.gpu


def _ptr(t):
  return ctypes.c_void_p(t.data_ptr())


def _qkv(rows, E, Hq, Hkv, D, scratch_offset):
  """Queries, keys and values of `rows` random rows through mtx_qkv_rope_append, its scratch so many bytes behind an allocation's start."""
  lib = _lib.load()
  g = torch.Generator(device="cuda").manual_seed(rows + E)
  rn = lambda *shape: torch.randn(*shape, generator=g, device="cuda").to(torch.bfloat16)
  x, w = rn(256, E), rn((Hq + 2 * Hkv) * D, E) / E**0.5
  T = 40
  pos, row = (torch.randint(0, hi, (rows,), generator=g, device="cuda").to(torch.int32) for hi in (3000, T))
  plane = torch.arange(rows, device="cuda", dtype=torch.int32)
  k, v = (torch.zeros(rows, Hkv, T, D, dtype=torch.bfloat16, device="cuda") for _ in range(2))
  q = torch.zeros(rows, Hq * D, dtype=torch.bfloat16, device="cuda")
  scratch = torch.empty(lib.mtx_qkv_rope_append_scratch_bytes(rows, D) + 256, dtype=torch.uint8, device="cuda")[scratch_offset:]
  stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
  _lib.check(lib.mtx_qkv_rope_append(_ptr(x), _ptr(w), _ptr(pos), _ptr(plane), _ptr(row), _ptr(q), _ptr(k), _ptr(v), rows, E, Hq, Hkv, D, T, 1.0, 10000.0, _ptr(scratch), stream))
  torch.cuda.synchronize()
  return q, k, v


@pytest.mark.parametrize("rows,E,Hq,Hkv,D", [(5, 256, 4, 2, 64), (65, 512, 4, 2, 64), (200, 512, 8, 8, 128), (256, 64, 20, 4, 64)])
def test_scratch_of_eight_byte_alignment(rows, E, Hq, Hkv, D):
  """The table of angles in the caller's scratch holds pairs of floats: any address that suits them will do, in every plan of the projection."""
  assert all(torch.equal(a, b) for a, b in zip(_qkv(rows, E, Hq, Hkv, D, 0), _qkv(rows, E, Hq, Hkv, D, 8)))
