"""The framework's settings for its matrix products hold for the products inside the nodes too."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

CODE = r'''
import glob
import torch
from pcf_nat_b200 import NAttention, block
from pcf_nat_b200.model import NABlock

torch.manual_seed(0)
layer = NAttention(40, 64, 2, 7, layout="channels_last").cuda()
stage = torch.nn.ModuleList([NABlock(40, 64, 2, 7, 4, "fused")]).cuda()
x = torch.randn(2, 40, 64, device="cuda").bfloat16()

def gradients(module):
    leaf = x.clone().requires_grad_()
    with torch.autocast("cuda", dtype=torch.bfloat16):
        y = layer(leaf * 1) if module is layer else block.run_blocks(stage, leaf * 1, None)
    return torch.autograd.grad(y, [leaf] + [p for n, p in module.named_parameters() if "relative" not in n], torch.ones_like(y))

want = [gradients(m) for m in (layer, stage)]

def close(got):
    return all(float((a.double() - b.double()).norm()) <= 2 * 2.0 ** -8 * float(b.double().norm()) for g, w in zip(got, want) for a, b in zip(g, w))

# each setting leaves the products to the framework, whose result is the same up to the order of sums
torch.backends.cuda.preferred_blas_library("cublaslt")
assert close([gradients(m) for m in (layer, stage)])
torch.backends.cuda.matmul.allow_bf16_reduced_precision_reduction = (False, False)      # (no split sums: with that library only)
assert close([gradients(m) for m in (layer, stage)])
torch.backends.cuda.matmul.allow_bf16_reduced_precision_reduction = (True, True)
torch.backends.cuda.preferred_blas_library("cublas")
torch.use_deterministic_algorithms(True)
assert close([gradients(m) for m in (layer, stage)])
torch.use_deterministic_algorithms(False)
assert all(torch.equal(a, b) for m, w in zip((layer, stage), want) for a, b in zip(gradients(m), w))
# products that could be tuned are noted down by the framework when they run
torch.cuda.tunable.enable(True)
torch.cuda.tunable.tuning_enable(False)
torch.cuda.tunable.record_untuned_enable(True)
for m in (layer, stage):
    before = sum(1 for f in glob.glob("untuned*") for _ in open(f))
    assert close([gradients(m)] if m is layer else [gradients(layer), gradients(m)])
    assert sum(1 for f in glob.glob("untuned*") for _ in open(f)) > before, m
print("ok")
'''


def test_settings_in_a_fresh_process(tmp_path):
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    env = dict(os.environ, PYTHONPATH=root + os.pathsep + os.environ.get("PYTHONPATH", ""), CUBLAS_WORKSPACE_CONFIG=":4096:8",
               PYTORCH_TUNABLEOP_UNTUNED_FILENAME=str(tmp_path / "untuned.csv"))
    r = subprocess.run([sys.executable, "-c", CODE], cwd=tmp_path, env=env, capture_output=True, text=True, timeout=600)
    assert r.returncode == 0 and "ok" in r.stdout, r.stdout[-2000:] + r.stderr[-2000:]
