"""na1d_fused_backward leaves delta_ws alone where na1d_fused_backward_workspace_floats says that it needs none."""
import random

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("seed", range(40))
def test_workspace_that_is_not_needed_is_not_touched(seed):
    from pcf_nat_b200 import _lib
    L, rng = _lib.lib(), random.Random(seed)
    C, heads, win, dil = rng.choice([8, 16, 24, 32, 48, 64, 96, 128, 192]), rng.choice([1, 2, 4, 16]), rng.randrange(3, 60), rng.choice([1, 1, 2, 3])
    T, batch, bias, grad = rng.randrange(20, 400), rng.randrange(1, 5), rng.random() < 0.6, rng.random() < 0.6
    left, N = rng.randrange(win), batch * heads
    if heads * win * 4 > 48 * 1024:
        pytest.skip("refused")
    q, k, v, d_o = (torch.randn(N, T, C, device="cuda").bfloat16() for _ in range(4))
    rpb = torch.randn(heads, win, device="cuda") if bias or grad else None
    o, lse = torch.empty_like(q), torch.empty(N, T, device="cuda")
    dq, dk, dv = (torch.empty_like(q) for _ in range(3))
    d_rpb = torch.zeros(heads, win, device="cuda") if grad else None
    p = lambda t: None if t is None else t.data_ptr()
    st = torch.cuda.current_stream().cuda_stream
    args = (N, heads, T, C, win, left, dil)
    _lib.check(L.na1d_fused_forward(p(o), p(lse), p(q), p(k), p(v), p(rpb), None, *args, C ** -0.5, _lib.NA1D_BF16, st), "na1d_fused_forward")
    floats = L.na1d_fused_backward_workspace_floats(*args, _lib.NA1D_BF16, int(rpb is not None), int(grad))
    route = L.na1d_fused_kernel_route(*args, _lib.NA1D_BF16, 1, int(rpb is not None), int(grad))
    assert floats in (0, N * T) and (floats == N * T if route == 0 else True) and (floats == 0 if route in (3, 4) else True)
    work = torch.full((N, T), 5.0, device="cuda")
    _lib.check(L.na1d_fused_backward(p(dq), p(dk), p(dv), p(d_rpb), p(d_o), p(q), p(k), p(v), p(o), p(lse), p(rpb), None, p(work), *args, C ** -0.5,
                                     _lib.NA1D_BF16, st), "na1d_fused_backward")
    assert floats or bool((work == 5.0).all())
