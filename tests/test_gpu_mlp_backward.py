"""Backward of a block's MLP in one kernel (na1d_mlp_backward) against the same formula in 64 bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu
D = 256


def _backward(d, f, w1, w2):
    from pcf_nat_b200 import _lib
    L, rows, n = _lib.lib(), f.shape[0], f.shape[1]
    floats = L.na1d_mlp_scratch_floats(rows, D, n)
    scratch = torch.full((floats + 4,), float("nan"), device="cuda")
    dh, df, g = (torch.full((rows + 1, k), 7.0, device="cuda", dtype=f.dtype) for k in (D, n, n))
    _lib.check(L.na1d_mlp_backward(dh.data_ptr(), df.data_ptr(), g.data_ptr(), d.data_ptr(), f.data_ptr(), w1.data_ptr(), w2.data_ptr(), scratch.data_ptr(), rows,
                                   D, n, _lib.NA1D_BF16 if f.dtype == torch.bfloat16 else _lib.NA1D_FP16, torch.cuda.current_stream().cuda_stream),
               "na1d_mlp_backward")
    assert L.na1d_device_status() == 0
    assert all(bool((t[rows:] == 7.0).all()) for t in (dh, df, g))
    return dh[:rows], df[:rows], g[:rows]


# rows: within one CTA, one pair of CTAs and beside them; a full round of the 74 pairs and one row more (its tile then split over the
# hidden layer); hidden sizes of one piece, of a number that splits unevenly, the usual one and the largest
@pytest.mark.parametrize("rows,hidden", [(1, 128), (127, 256), (129, 1024), (256, 128), (257, 1280), (1000, 640), (18944, 128), (18945, 1024), (38400, 1024)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_mlp_backward(rows, hidden, dtype):
    gen = torch.Generator(device="cuda").manual_seed(rows + hidden)
    rn = lambda *s: torch.randn(*s, device="cuda", generator=gen)
    d, f, w1, w2 = rn(rows, D).to(dtype), (2 * rn(rows, hidden)).to(dtype), (rn(hidden, D) / 16).to(dtype), (rn(D, hidden) * hidden ** -0.5).to(dtype)
    x, dd, a1, a2 = f.double(), d.double(), w1.double(), w2.double()
    cdf = torch.special.ndtr(x)
    slope = cdf + x * torch.exp(-x * x / 2) * (2 * torch.pi) ** -0.5
    g = x * cdf
    dg = dd @ a2
    df = dg * slope
    dh = df @ a1
    u = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11     # relative rounding to 16 bits: half a unit of 8 or 11 digits
    got_h, got_f, got_g = _backward(d, f, w1, w2)
    # Phi(-|x|) is off by 8e-7 at most and the density by less; results are rounded once (3e-8: half the smallest fp16); sums of 256 and
    # of `hidden` products in 32 bits
    assert bool(((got_g.double() - g).abs() <= u * g.abs() + 1e-6 * x.abs() + 3e-8).all())
    off = u * df.abs() + 2e-6 * dg.abs() + slope.abs() * (dd.abs() @ a2.abs()) * 2.0 ** -16 + 3e-8
    assert bool(((got_f.double() - df).abs() <= off).all())
    assert bool(((got_h.double() - dh).abs() <= off @ a1.abs() + u * dh.abs() + (df.abs() @ a1.abs()) * 2.0 ** -14 + 3e-8).all())
    # no further off than the products with the gradient of the hidden layer rounded in between
    passes = ((d @ w2).double() * slope).to(dtype)
    assert float((got_f.double() - df).norm()) <= float((passes.double() - df).norm()) * 1.02
    assert float((got_h.double() - dh).norm()) <= float(((passes @ w1).double() - dh).norm()) * 1.02
    assert all(torch.equal(a, b) for a, b in zip(_backward(d, f, w1, w2), (got_h, got_f, got_g)))


def test_gelu_and_slope_of_every_16_bit_value():
    """The hidden layer over all finite fp16 values and the special ones, through an identity in place of the weights."""
    x = torch.arange(-32768, 32768, device="cuda", dtype=torch.int32).to(torch.int16).view(torch.float16)
    x = x[torch.isfinite(x)]
    f = torch.zeros(256, 256, device="cuda", dtype=torch.float16).view(-1)
    f[:x.numel()] = x
    f[-3:] = torch.tensor([float("inf"), 300.0, float("nan")], dtype=torch.float16)
    f = f.view(256, 256)
    one = torch.ones(256, D, device="cuda", dtype=torch.float16)
    eye = torch.eye(256, device="cuda", dtype=torch.float16)
    _, df, g = _backward(one, f, eye, eye)
    xd = f.double()
    value = xd * torch.special.ndtr(xd)
    slope = torch.special.ndtr(xd) + xd * torch.exp(-xd * xd / 2) * (2 * torch.pi) ** -0.5
    ok = torch.isfinite(xd)
    assert bool(((g.double() - value).abs()[ok] <= 2.0 ** -11 * value.abs()[ok] + 1e-6 * xd.abs()[ok].clamp(max=8) + 3e-8).all())
    assert bool(((df.double() - slope).abs()[ok] <= 2.0 ** -11 * slope.abs()[ok] + 2e-6 + 3e-8).all())
    assert float(g.view(-1)[-3]) == float("inf") and float(g.view(-1)[-2]) == 300.0 and bool(torch.isnan(g.view(-1)[-1])) and bool(torch.isnan(df.view(-1)[-1]))


def test_refused():
    from pcf_nat_b200 import _lib
    L = _lib.lib()
    t = torch.zeros(1 << 20, device="cuda", dtype=torch.float16)
    p = t.data_ptr()
    st = torch.cuda.current_stream().cuda_stream
    call = lambda dh=p, df=p, f=p, scratch=p, rows=100, D_=D, F=512: L.na1d_mlp_backward(dh, df, p, p, f, p, p, scratch, rows, D_, F, _lib.NA1D_FP16, st)
    for bad in (dict(F=192), dict(F=1408), dict(D_=128), dict(rows=0), dict(dh=p + 16), dict(df=p + 16), dict(f=p + 16), dict(scratch=None), dict(df=None)):
        assert call(**bad) != 0


@pytest.mark.parametrize("chained", [False, True])
def test_second_derivative_of_blocks_with_one_output(chained):
    """As for the blocks of other sizes: a gradient penalty through the node gives what the modules give (eight rounding steps of bf16)."""
    from pcf_nat_b200 import block
    from pcf_nat_b200.model import NABlock
    torch.manual_seed(0)
    st = torch.nn.ModuleList(NABlock(40, D, 4, 7, 4, "fused") for _ in range(2 if chained else 1)).cuda()
    for n, p in st.named_parameters():
        p.requires_grad_("norm1.bias" not in n and "fc1.weight" not in n and "fc2.bias" not in n)
    params = [p for p in st.parameters() if p.requires_grad]
    got, first = {}, {}
    for kind in ("node", "modules"):
        x = (0.5 * torch.randn(2, 40, D, device="cuda", generator=torch.Generator(device="cuda").manual_seed(1))).to(torch.bfloat16).requires_grad_()
        with torch.autocast("cuda", dtype=torch.bfloat16):
            y = block.run_blocks(st, 2 * x, None) if kind == "node" else 2 * x
            for b in st if kind == "modules" else ():
                y = b(y)
        first[kind] = torch.autograd.grad(y.float().pow(2).sum(), [x] + params, retain_graph=True)
        g, = torch.autograd.grad(y.float().pow(2).sum(), x, create_graph=True)
        out = torch.autograd.grad(g.float().pow(2).sum(), [x] + params, allow_unused=True)
        got[kind] = [g.detach()] + [torch.zeros_like(p) if o is None else o for o, p in zip(out, [x] + params)]
    for r in (got, first):
        for a, b in zip(r["node"], r["modules"]):
            assert a.dtype == b.dtype and float((a.double() - b.double()).norm()) <= 8 * 2.0 ** -8 * float(b.double().norm()) + 1e-6
