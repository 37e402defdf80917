"""Parameter gradients of projections: distance from 64 bits, against sums in fp32 by other means."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mean", [0.0, 1.0])
@pytest.mark.parametrize("rows,M,N", [(300, 1024, 256), (2400, 256, 1024), (9600, 256, 256), (38400, 1024, 256), (38400, 256, 256), (38401, 264, 520)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_no_further_off_than_other_sums_in_fp32(rows, M, N, dtype, mean):
    """The weight gradient against the library's product with fp32 sums, the bias gradient against a pass of column sums. Both sides are off
    by rounding errors of sums in different orders, averaged over hundreds of results: half as much again is allowed, a third for the
    bias, whose sums both round to nearest."""
    import block_passes
    from test_gpu_wgrad import _gradients
    g = torch.Generator(device="cuda").manual_seed(rows)
    dy, x = ((torch.randn(rows, k, device="cuda", generator=g) + mean).to(dtype) for k in (M, N))
    (w,), (b,) = _gradients([(dy, x)], True)
    rw, rb = dy.double().t() @ x.double(), dy.double().sum(0)
    far = lambda a, r: float((a.double() - r).norm() / r.norm())
    assert far(w, rw) <= 1.5 * far(torch.mm(dy.t(), x, out_dtype=torch.float32), rw)
    assert far(b, rb) <= 4 / 3 * far(block_passes.column_sums(dy, block_passes.scratch_for(rows, M, M, dy.device)), rb)
