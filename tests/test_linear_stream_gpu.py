"""Products of few rows (csrc/linear_stream.cuh): the bfloat16 engine against the same engine with the kernel switched off (linear_mma_kernel, whose bits
it claims) and against the float32 engine, whose projections are fp32 FMA kernels, with the same weights.  Rows at the edges of its 16- and
32-row parts, k of one stage and of more than the ring holds, output widths that leave the last tile of columns part empty, experts with none to
a few tokens."""

import os
import subprocess
import sys

import numpy as np
import pytest
import torch

from maxtext_indextts2_b200 import kifusun, maxengine, pyconfig, zakelorn

pytestmark = pytest.mark.gpu

NAMES = ("kifusun", "zakelorn")
SIZES = [(64, 1), (192, 16), (192, 17), (640, 31), (640, 32), (192, 33)]


def _model(name, width):
  if name == "kifusun":
    return kifusun, kifusun.model_dict(width, 333, [kifusun.attention_layer(2, 1, 32, 32, 64, ff=192, bias_max=64.0)] * 2)
  ffs = [zakelorn.moe_ff(7, 2, 128, identity=1, shared_ff=64), zakelorn.moe_ff(40, 3, 64, identity=2)]
  return zakelorn, zakelorn.model_dict(width, 333, [zakelorn.parallel_layer(zakelorn.attention_part(2, 1, 32, window=64, keep_first=4), zakelorn.lightning_part(2, 32), mlp=f)
                                                    for f in ffs])


def _logits(name, width, rows, dtype):
  design, model = _model(name, width)
  toks = np.random.Generator(np.random.PCG64(rows)).integers(0, model["vocab"], size=rows).tolist()
  cfg = pyconfig.from_model_dict(model, dtype=dtype, per_device_batch_size=2, max_target_length=64, pagedattn_tokens_per_page=16, pagedattn_num_pages=12)
  engine = maxengine.MaxEngine(cfg)
  engine.load_params(design.random_tensors(cfg, seed=3))
  engine.init_decode_state()
  return engine.step([(0, toks, list(range(rows)))]).cpu()


def dump(path):
  torch.save({(n, w, r): _logits(n, w, r, "bfloat16") for n in NAMES for w, r in SIZES}, path)


@pytest.fixture(scope="module")
def switched_off(tmp_path_factory):  # (the switch is read once per process)
  path = str(tmp_path_factory.mktemp("linear") / "logits.pt")
  root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
  subprocess.run([sys.executable, "-c", f"from tests.test_linear_stream_gpu import dump; dump({path!r})"], cwd=root, check=True, timeout=300,
                 env=dict(os.environ, MTX_LINEAR_STREAM="0"))
  return torch.load(path)


@pytest.mark.parametrize("name", NAMES)
@pytest.mark.parametrize("width,rows", SIZES)
def test_few_rows(name, width, rows, switched_off):
  got, want = _logits(name, width, rows, "bfloat16"), _logits(name, width, rows, "float32").double()
  assert torch.equal(got, switched_off[name, width, rows])
  off = (got.double() - want).square().mean(1).sqrt() / want.square().mean().sqrt()
  # bf16 operands (2^-9 each) through two layers: the designs' own tests allow 3e-2; a routed row whose experts are a near-tie may be further off
  # than that (its bits are compared above)
  assert float(off.max() if name == "kifusun" else off.median()) < 3e-2
