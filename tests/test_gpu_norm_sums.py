"""LayerNorm's backward in rows, and the column sums of two of them in one launch, against the pass that does both."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("rows,D", [(1, 8), (9, 264), (5000, 256), (33, 1024)])
def test_two_passes_and_their_sums(rows, D, dtype):
    from pcf_nat_b200 import _lib
    L, st = _lib.lib(), torch.cuda.current_stream().cuda_stream
    code = _lib.NA1D_BF16 if dtype == torch.bfloat16 else _lib.NA1D_FP16
    gen = torch.Generator(device="cuda").manual_seed(rows + D)
    rn = lambda *s: torch.randn(*s, device="cuda", generator=gen)
    room = (L.na1d_block_scratch_floats(rows, D, 8) + 3) // 4 * 4
    parts, got, want, dx = torch.full((2 * room,), float("nan"), device="cuda"), torch.full((2, 3, D), float("nan"), device="cuda"), [], []
    for k in range(2):
        dy, x, w = rn(rows, D).to(dtype), rn(rows, D).to(dtype), rn(D)
        mean, rstd = x.float().mean(1), 1 / (x.float().std(1, unbiased=False) + 0.1)
        sums, one, two = torch.empty(3, D, device="cuda"), torch.empty_like(x), torch.empty_like(x)
        scratch = torch.empty(room, device="cuda")
        _lib.check(L.na1d_layer_norm_backward(one.data_ptr(), sums.data_ptr(), scratch.data_ptr(), dy.data_ptr(), x.data_ptr(), mean.data_ptr(), rstd.data_ptr(),
                                              w.data_ptr(), None, rows, D, code, st), "both")
        _lib.check(L.na1d_layer_norm_backward_rows(two.data_ptr(), parts[k * room:].data_ptr(), dy.data_ptr(), x.data_ptr(), mean.data_ptr(), rstd.data_ptr(),
                                                   w.data_ptr(), None, rows, D, code, st), "rows")
        assert torch.equal(one, two)
        want.append(sums)
    _lib.check(L.na1d_layer_norm_sums(got[0].data_ptr(), got[1].data_ptr(), parts.data_ptr(), parts[room:].data_ptr(), rows, D, st), "sums")
    assert torch.equal(got, torch.stack(want))
    assert L.na1d_layer_norm_sums(got.data_ptr(), None, parts.data_ptr(), parts.data_ptr(), rows, D, st) != 0
    assert L.na1d_layer_norm_backward(one.data_ptr(), None, scratch.data_ptr(), dy.data_ptr(), x.data_ptr(), mean.data_ptr(), rstd.data_ptr(), w.data_ptr(), None,
                                      rows, D, code, st) != 0
