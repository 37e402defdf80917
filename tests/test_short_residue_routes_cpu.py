"""The rule that takes dilated calls with short residues from the segmented tiling (a host-only query)."""
import pytest
import torch

from pcf_nat_b200 import ops


# (channels, tokens, dilation, window) -> kernels of the backward: 2 = segmented tiling, 0 or 3 = general
@pytest.mark.parametrize("C,T,dil,win,segmented", [
    (32, 24, 2, 27, True), (32, 36, 3, 33, True), (32, 24, 2, 22, False), (32, 20, 2, 23, True), (32, 18, 2, 27, False), (32, 24, 2, 17, False), (32, 36, 3, 15, False),
    (64, 36, 3, 15, False), (64, 39, 3, 15, True), (64, 48, 3, 9, False), (64, 51, 3, 9, True)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_backward(C, T, dil, win, segmented, dtype):
    assert (ops.kernel_route(4000, 4, T, C, win, win // 2, dil, dtype, True, True, True) == 2) == segmented
