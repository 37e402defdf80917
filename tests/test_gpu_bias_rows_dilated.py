"""NA1D_BIAS_GRAD_ROWS=1 for dilated calls with short residues: the bias gradient keeps its fixed order of sums."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

CODE = r'''
import sys, torch
sys.path[:0] = ["tests", "tests/golden"]
from gpu_util import assert_close
from oracle import na1d_oracle as orc
from pcf_nat_b200 import ops
for C, T, win, dil in ((64, 36, 7, 3), (32, 33, 15, 3), (64, 48, 9, 3), (64, 49, 9, 3)):
    N, H, left, sc = 1200, 4, win // 2, C ** -0.5
    g = torch.Generator().manual_seed(T)
    q, k, v, d_o = ((torch.randn(N, T, C, generator=g) * C ** -0.25).to(torch.bfloat16) for _ in range(4))
    rpb = 0.3 * torch.randn(H, win, generator=g)
    assert ops.kernel_route(N, H, T, C, win, left, dil, q.dtype, True, True, True) == 2
    o, lse = ops.fused_forward(q.cuda(), k.cuda(), v.cuda(), win, left, dil, sc, rpb.cuda(), None, H)
    args = (d_o.cuda(), q.cuda(), k.cuda(), v.cuda(), o, lse, win, left, dil, sc, rpb.cuda(), None, H)
    a = [ops.fused_backward(*args, need_d_rpb=True)[3] for _ in range(4)]
    ops.device_status()
    if C == 64:      # (32 channels: one shared atomic per lane and tile)
        assert all(torch.equal(a[0], b) for b in a[1:])
    ref = orc.na1d_fused_with_grads(q.float(), k.float(), v.float(), d_o.float(), win, left, dilation=dil, scale=sc, rpb=rpb, heads=H)[4]
    assert_close(a[0], ref, torch.bfloat16, "drpb", factor=2.0)
    # without a bias gradient the route is the cheaper one
    assert ops.kernel_route(N, H, T, C, win, left, dil, q.dtype, True, True, False) == ops.kernel_route(N, H, T, C, win, left, dil, q.dtype, True)
print("ok")
'''


def test_short_residues_keep_the_order_of_sums():
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    env = dict(os.environ, NA1D_BIAS_GRAD_ROWS="1", PYTHONPATH=root + os.pathsep + os.environ.get("PYTHONPATH", ""))
    r = subprocess.run([sys.executable, "-c", CODE], cwd=root, env=env, capture_output=True, text=True, timeout=600)
    assert r.returncode == 0 and "ok" in r.stdout, r.stdout[-2000:] + r.stderr[-2000:]
