"""The marching kernels (16-channel rows) against plain PyTorch in 64 bits: windows at the edges of their two and three key
tiles, one-sided windows, sequences around a block of 16 and a strip, dilations with empty and uneven residues, padding, dense
and packed layouts, strips that own part of a sequence, the bias gradient across heads."""
import pytest
import torch

from test_gpu_mma import _inputs, _reference, _run

pytestmark = pytest.mark.gpu

#      B  H  T    C   win left dil bias  padded
CASES = [
    (1, 1, 1, 16, 1, 0, 1, True, False),
    (2, 3, 16, 16, 17, 8, 1, True, True),
    (1, 2, 17, 16, 17, 16, 1, False, True),
    (2, 5, 150, 16, 27, 13, 1, True, True),
    (3, 2, 150, 16, 33, 32, 1, True, False),
    (1, 3, 97, 16, 33, 0, 1, True, True),
    (2, 2, 64, 16, 18, 3, 2, True, True),
    (2, 1, 5, 16, 9, 4, 7, True, True),          # more residues than tokens
    (1, 40, 63, 16, 7, 3, 3, True, False),        # more heads than the tcgen05 kernels take
    (1, 1, 3000, 16, 15, 7, 1, True, True),       # several strips per sequence
    (1, 2, 1111, 16, 33, 20, 2, True, True),
    (300, 1, 33, 16, 2, 1, 1, True, False),
    (2, 3, 150, 32, 27, 13, 1, True, True),       # forward only: the backward of 32 channels is another family's
    (1, 2, 700, 32, 9, 8, 3, True, False),
    (2, 1, 15, 32, 33, 0, 1, False, True),
]
EPS = {torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11}


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("case", CASES)
def test_against_64_bits(case, dtype):
    """Probabilities, dS and results are each rounded to 16 bits once (half a step, random): the 2-norm error of a result stays
    below one step of the largest of the three, 1.2 for the few elements of a bias gradient."""
    from pcf_nat_b200 import ops
    args = _inputs(case, dtype)
    got, again = _run(ops.FAMILY_MARCH, case, *args), _run(ops.FAMILY_MARCH, case, *args)
    for i, (a, r) in enumerate(zip(got, _reference(case, *args))):
        assert float((a.double() - r).norm()) <= 1.2 * EPS[dtype] * float(r.norm()) + 1e-6, i
        if i < 4:
            assert torch.equal(a, again[i]), i            # one owner per result: the same bits from run to run
            assert float((a.double() - r).abs().max()) <= 4 * EPS[dtype] * float(r.abs().max()) + 1e-5, i


@pytest.mark.parametrize("T,win,left,dil,C", [(150, 27, 13, 1, 16), (64, 9, 8, 3, 16), (331, 33, 16, 1, 16), (150, 27, 13, 1, 32)])
def test_packed_layout_and_automatic_route(T, win, left, dil, C):
    """The automatic route of dense and packed calls is the marching one, with the same bits in both layouts."""
    from pcf_nat_b200 import ops
    B, H = 3, 5
    g = torch.Generator(device="cuda").manual_seed(3)
    qkv = torch.randn(B, T, 3, H, C, device="cuda", generator=g).bfloat16()
    d = torch.randn(B, T, H, C, device="cuda", generator=g).bfloat16()
    rpb = torch.randn(H, win, device="cuda", generator=g)
    vl = torch.tensor([T, T // 2, 3], device="cuda", dtype=torch.int32)
    leaf = qkv.view(B, T, 3 * H * C).clone().requires_grad_()
    bias = rpb.clone().requires_grad_()
    y = ops.na1d_fused_packed(leaf, H, win, left, dil, 0.25, bias, vl)
    dx, db = torch.autograd.grad(y, (leaf, bias), d.view(B, T, H * C))
    q, k, v = (qkv[:, :, i].permute(0, 2, 1, 3).reshape(B * H, T, C).contiguous() for i in range(3))
    dd = d.permute(0, 2, 1, 3).reshape(B * H, T, C).contiguous()
    for family in (ops.FAMILY_MARCH, ops.FAMILY_AUTO):
        old = ops.set_kernel_family(family)
        try:
            o, lse = ops.fused_forward(q, k, v, win, left, dil, 0.25, rpb, vl, H)
            grads = ops.fused_backward(dd, q, k, v, o, lse, win, left, dil, 0.25, rpb, vl, H, need_d_rpb=True)
        finally:
            ops.set_kernel_family(old)
        assert torch.equal(o.view(B, H, T, C).permute(0, 2, 1, 3).reshape(B, T, H * C), y)
        if C != 16:
            continue                              # (the backward of 32 channels is another family's, with another tiling in each layout)
        for i in range(3):
            assert torch.equal(grads[i].view(B, H, T, C).permute(0, 2, 1, 3), dx.view(B, T, 3, H, C)[:, :, i]), i
        assert torch.allclose(grads[3], db, rtol=1e-4, atol=1e-4)


def test_strips_leave_no_seam():
    """One long sequence (strips of a few blocks) and the same rows inside a batch large enough for whole-sequence strips."""
    from pcf_nat_b200 import ops
    case = (1, 1, 700, 16, 33, 9, 1, True, False)
    q, k, v, d_o, rpb, _ = _inputs(case, torch.bfloat16)
    one = _run(ops.FAMILY_MARCH, case, q, k, v, d_o, rpb, None)
    many = _run(ops.FAMILY_MARCH, (4000,) + case[1:], *(t.expand(4000, 700, 16).contiguous() for t in (q, k, v, d_o)), rpb, None)
    for i in range(4):
        assert torch.equal(many[i][0], one[i][0]) and torch.equal(many[i][3999], one[i][0])
    assert torch.allclose(many[4] / 4000, one[4], rtol=1e-3, atol=1e-3)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_segmented_tiling_where_the_marching_kernels_stand_for_it(dtype):
    """The tcgen05 kernels on the segmented tiling at the sizes of their own test that the automatic choice gives to the marching
    ones in some calls and to them in others: forward and backward against 64 bits."""
    from test_gpu_segmented import SEG_SHAPES

    from pcf_nat_b200 import ops
    for N, H, T, C, win, left, dil in SEG_SHAPES:
        if C == 64:
            continue
        case = (N // H, H, T, C, win, left, dil, True, True)
        args = _inputs(case, dtype)
        march = _run(ops.FAMILY_MARCH, case, *args)
        got = _run(ops.FAMILY_SEGMENTED_ONLY, case, *args)
        assert not torch.equal(march[0], got[0]) or T < 32, case           # (another kernel)
        for i, (a, r) in enumerate(zip(got, _reference(case, *args))):
            assert float((a.double() - r).norm()) <= 1.2 * EPS[dtype] * float(r.norm()) + 1e-6, (case, i)
