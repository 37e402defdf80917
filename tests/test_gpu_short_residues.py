"""The kernels that short residues and 32-channel rows are given against the ones they had, and against the oracle's formula."""
import pytest
import torch

from gpu_util import assert_close, assert_close_strict
from oracle import na1d_oracle as orc

pytestmark = pytest.mark.gpu


# (channels, sequences, tokens, window, dilation): residues on both sides of 12, 16 and 40 rows; 32-channel dense forwards above 2^18
# rows on both sides of 256 tokens, and dilated ones
@pytest.mark.parametrize("C,N,T,win,dil", [
    (64, 8, 36, 7, 3), (64, 8, 37, 7, 3), (64, 8, 120, 9, 3), (64, 8, 123, 9, 3), (64, 8, 48, 9, 3), (64, 8, 49, 11, 3), (64, 4, 96, 15, 3), (32, 8, 33, 5, 3),
    (32, 8, 36, 15, 3), (32, 8, 48, 9, 3), (32, 2800, 97, 9, 1), (32, 1040, 255, 27, 1), (32, 1040, 256, 27, 1), (32, 1300, 211, 5, 2), (32, 2100, 130, 9, 3)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_routes(C, N, T, win, dil, dtype):
    from pcf_nat_b200 import _lib, na1d_fused
    L, H, left = _lib.lib(), 4, win // 2
    g = torch.Generator().manual_seed(C + T + win)
    q, k, v, d = ((torch.randn(N, T, C, generator=g)).to(dtype).cuda() for _ in range(4))
    rpb = (0.1 * torch.randn(H, win, generator=g)).cuda()

    def run():
        leaves = [t.detach().requires_grad_(True) for t in (q, k, v, rpb)]
        o = na1d_fused(leaves[0], leaves[1], leaves[2], win, left, dil, C ** -0.5, leaves[3], None, H)
        return [o.detach()] + list(torch.autograd.grad(o, leaves, d))

    got = run()
    code = _lib.NA1D_BF16 if dtype == torch.bfloat16 else _lib.NA1D_FP16
    tp = (T + dil - 1) // dil
    route = [L.na1d_fused_kernel_route(N, H, T, C, win, left, dil, code, b, 1, 1) for b in (0, 1)]
    if C == 32:
        assert route[0] == (1 if dil == 1 and T < 256 else 4)
    elif tp <= 40:
        assert route[0] in (0, 3)
    if dil == 3 and (tp <= 12 or (tp <= 16 and win <= 9)):
        assert route[1] in (0, 3)
    # whole sequences against the oracle
    n = min(N, 8)
    ref = orc.na1d_fused_with_grads(*(t[:n].float().cpu() for t in (q, k, v, d)), win, left, dilation=dil, scale=C ** -0.5, rpb=rpb.cpu(), heads=H)
    assert_close_strict(got[0][:n], ref[0], dtype, "o")
    for a, b, what in zip(got[1:4], ref[1:4], ("dq", "dk", "dv")):
        assert_close(a[:n], b, dtype, what)
    # everything against the tcgen05 kernels
    old = L.na1d_set_kernel_family(5 if dil > 1 else 1)
    try:
        other = run()
    finally:
        L.na1d_set_kernel_family(old)
    for a, b, what in zip(got[:4], other[:4], ("o", "dq", "dk", "dv")):
        assert_close(a, b.float(), dtype, what)
    # the bias gradient sums N T / H values of dS, each rounded to 16 bits on one side at most: 2^-8 or 2^-11 of |dS| < 8, as a random walk
    # (six standard deviations)
    step = 8 * 2.0 ** (-8 if dtype == torch.bfloat16 else -11)
    assert float((got[4] - other[4]).abs().max()) <= 6 * step * (N / H * T) ** 0.5
