"""A block's MLP in one kernel (na1d_mlp_forward) against the same formula in 64 bits."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu
D = 256


def _inputs(rows, hidden, dtype, scale=1.0):
    g = torch.Generator(device="cuda").manual_seed(rows + hidden)
    rn = lambda *s: torch.randn(*s, device="cuda", generator=g)
    return (rn(rows, D).to(dtype), (scale * rn(rows, D)).to(dtype), (rn(hidden, D) / 16).to(dtype), 0.3 * rn(hidden), (rn(D, hidden) * hidden ** -0.5).to(dtype),
            0.3 * rn(D))


def _mlp(s, h, w1, b1, w2, b2, hidden_layer, ld=D):
    from pcf_nat_b200 import _lib
    L, rows, n = _lib.lib(), s.shape[0], w1.shape[0]
    floats = L.na1d_mlp_scratch_floats(rows, D, n)
    assert floats >= 0
    scratch = torch.full((floats + 4,), float("nan"), device="cuda")
    out = torch.full((rows + 1, ld), 7.0, device="cuda", dtype=s.dtype)
    f = torch.full((rows + 1, n), 7.0, device="cuda", dtype=s.dtype) if hidden_layer else None
    _lib.check(L.na1d_mlp_forward(out.data_ptr(), ld, None if f is None else f.data_ptr(), s.data_ptr(), h.data_ptr(), w1.data_ptr(), b1.data_ptr(),
                                  w2.data_ptr(), b2.data_ptr(), scratch.data_ptr(), rows, D, n, _lib.NA1D_BF16 if s.dtype == torch.bfloat16 else _lib.NA1D_FP16,
                                  torch.cuda.current_stream().cuda_stream), "na1d_mlp_forward")
    assert L.na1d_device_status() == 0
    assert bool((out[rows:] == 7.0).all()) and bool((out[:, D:] == 7.0).all()) and (f is None or bool((f[rows:] == 7.0).all()))
    return out[:rows, :D], None if f is None else f[:rows]


# rows: within one CTA, one pair of CTAs and beside them; a full round of the 74 pairs and one row more (its tile then split over the
# hidden layer); hidden sizes of one piece, of a number that splits unevenly, the usual one and the largest
@pytest.mark.parametrize("rows,hidden", [(1, 128), (127, 256), (129, 1024), (256, 128), (257, 1280), (1000, 640), (18944, 128), (18945, 1024), (38400, 1024)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_mlp(rows, hidden, dtype):
    a = _inputs(rows, hidden, dtype)
    s, h, w1, b1, w2, b2 = (t.double() for t in a)
    f = h @ w1.t() + b1
    g = F.gelu(f)
    z = g @ w2.t() + b2
    ref = s + z
    u = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11     # relative rounding to 16 bits: half a unit of 8 or 11 digits
    out, hid = _mlp(*a, True)
    # the hidden layer is rounded once; GELU is off by 1.1e-5 of its argument at most and rounded once, z and the result once each;
    # 1e-5 and 3e-8 (half the smallest fp16) for sums in 32 bits and results below the normal range
    assert bool(((hid.double() - f).abs() <= u * f.abs() + 1e-5).all())
    bound = (u * g.abs() + 1.2e-5 * f.abs() + 3e-8) @ w2.abs().t() + u * (z.abs() + ref.abs()) * 1.01 + 1e-5
    assert bool(((out.double() - ref).abs() <= bound).all())
    # and no further off than the products and GELU as separate passes
    gg = F.gelu((a[1] @ a[2].t() + a[3].to(dtype)).float()).to(dtype)
    passes = (a[0].float() + (gg @ a[4].t() + a[5].to(dtype)).float()).to(dtype)
    assert float((out.double() - ref).norm()) <= 1.02 * float((passes.double() - ref).norm())
    # the same bits without the hidden layer, into wider rows, and again
    assert torch.equal(_mlp(*a, False)[0], out) and torch.equal(_mlp(*a, False, ld=3 * D + 8)[0], out)


def test_gelu_tail():
    """Large negative arguments: the tail keeps its relative accuracy (1e-4 up to 4, 1e-3 up to 6), nothing overflows beyond it."""
    x = torch.linspace(-30, 30, 1024, device="cuda")
    s = torch.zeros(256, D, device="cuda", dtype=torch.bfloat16)
    w1, w2 = torch.zeros(1024, D, device="cuda", dtype=torch.bfloat16), torch.zeros(D, 1024, device="cuda", dtype=torch.bfloat16)
    worst = []
    for k in range(0, 1024, D):      # the hidden layer is x (from the bias), the second product picks 256 of its columns
        w2.zero_()
        w2[torch.arange(D), k + torch.arange(D)] = 1
        got = _mlp(s, s, w1, x, w2, torch.zeros(D, device="cuda"), False)[0][0].double()
        xd = x[k:k + D].double()
        ref = xd * torch.special.ndtr(xd)
        assert bool(torch.isfinite(got).all())
        worst.append(((got - ref).abs() / ref.abs().clamp_min(1e-300), xd))
    err, xd = (torch.cat(t) for t in zip(*worst))
    near, mid, far = xd.abs() <= 4, (xd < -4) & (xd >= -6), xd < -13
    # rounded to bf16 twice (the hidden operand and z): 2 * 2^-8
    assert float(err[near | (xd > 4)].max()) <= 2 * 2.0 ** -8 + 1e-4 and float(err[mid].max()) <= 2 * 2.0 ** -8 + 1e-3
    assert bool(((err * (xd * torch.special.ndtr(xd)).abs())[far] <= 1e-30).all())


@pytest.mark.parametrize("D_,hidden", [(256, 1408), (256, 192), (128, 512)])
def test_sizes_that_are_refused(D_, hidden):
    from pcf_nat_b200 import _lib
    assert _lib.lib().na1d_mlp_scratch_floats(100, D_, hidden) == -1
