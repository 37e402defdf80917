"""LayerNorm by groups of four rows (large calls) and row by row (small ones): the same bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [32767, 32768, 32769, 65535, 65538])
@pytest.mark.parametrize("D", [8, 200, 256])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("add", [False, True])
def test_rows_of_a_large_call(rows, D, dtype, add):
    import block_passes
    g = torch.Generator(device="cuda").manual_seed(rows + D)
    rn = lambda *s: torch.randn(*s, device="cuda", generator=g)
    x, dx, w, b = rn(rows, D).to(dtype), rn(rows, D).to(dtype) if add else None, rn(D), rn(D)
    whole = block_passes.layer_norm(x, dx, w, b, 1e-5, True)
    for lo, hi in ((0, 1000), (rows - 1001, rows)):
        part = block_passes.layer_norm(x[lo:hi].clone(), dx[lo:hi].clone() if add else None, w, b, 1e-5, True)
        assert torch.equal(part[0], whole[0][lo:hi]) and torch.equal(part[1], whole[1][lo:hi])
        assert torch.equal(part[2][:hi - lo], whole[2][lo:hi]) and torch.equal(part[3][:hi - lo], whole[3][lo:hi])
