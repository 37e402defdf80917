"""A block's MLP in one kernel with the rounding points of its passes (na1d_mlp_forward_rounded): a network gives the values of the
passes one by one, in evaluation up to a rare 16-bit step where the library shares out a sum in another way."""
import pytest
import torch

pytestmark = pytest.mark.gpu
D, DT = 256, [torch.bfloat16, torch.float16]


def _rounded(s, h, w1, b1, w2, b2, hidden_layer, ld=D):
    from pcf_nat_b200 import _lib
    L, rows, n = _lib.lib(), s.shape[0], w1.shape[0]
    scratch = torch.full((L.na1d_mlp_scratch_floats(rows, D, n) + 4,), float("nan"), device="cuda") if hidden_layer else None
    out = torch.full((rows + 1, ld), 7.0, device="cuda", dtype=s.dtype)
    f = torch.full((rows + 1, n), 7.0, device="cuda", dtype=s.dtype) if hidden_layer else None
    _lib.check(L.na1d_mlp_forward_rounded(out.data_ptr(), ld, None if f is None else f.data_ptr(), s.data_ptr(), h.data_ptr(), w1.data_ptr(), b1.data_ptr(),
                                          w2.data_ptr(), b2.data_ptr(), None if scratch is None else scratch.data_ptr(), rows, D, n,
                                          _lib.NA1D_BF16 if s.dtype == torch.bfloat16 else _lib.NA1D_FP16, torch.cuda.current_stream().cuda_stream),
               "na1d_mlp_forward_rounded")
    assert L.na1d_device_status() == 0
    assert bool((out[rows:] == 7.0).all()) and bool((out[:, D:] == 7.0).all()) and (f is None or bool((f[rows:] == 7.0).all()))
    return out[:rows, :D], None if f is None else f[:rows]


def _passes(s, h, w1, b1, w2, b2):
    import block_passes
    f = torch.addmm(b1, h, w1.t())
    return s + torch.addmm(b2, block_passes.gelu(f), w2.t()), f


@pytest.mark.parametrize("rows,hidden", [(1, 128), (127, 256), (257, 1280), (1000, 640), (18945, 1024), (38400, 1024)])
@pytest.mark.parametrize("dtype", DT)
def test_values_of_the_passes(rows, hidden, dtype):
    g = torch.Generator(device="cuda").manual_seed(rows + hidden)
    rn = lambda *s: torch.randn(*s, device="cuda", generator=g)
    a = (rn(rows, D).to(dtype), rn(rows, D).to(dtype), (rn(hidden, D) / 16).to(dtype), (0.3 * rn(hidden)).to(dtype), (rn(D, hidden) * hidden ** -0.5).to(dtype),
         (0.3 * rn(D)).to(dtype))
    want, want_f = _passes(*a)
    out, _ = _rounded(*a, False)
    train, f = _rounded(*a, True)
    # sums of exact products in fp32 (2^-13 and 2^-16 of a 16-bit step between neighbouring ones): where they are made in another order, a few
    # of these steps lie between them, and 1 result in 1000 is rounded the other way. Rounding elsewhere, of the biases or
    # after GELU alone, would move a third of all values.
    for x, y in ((out, want), (train, want), (f, want_f)):
        differ = (x != y).double().mean()
        assert float(differ) <= 0.005 + 1 / x.numel()
        assert float((x.double() - y.double()).norm()) <= 1e-4 * float(y.double().norm()) + 1e-3 / rows ** 0.5
    assert torch.equal(_rounded(*a, False, ld=3 * D + 8)[0], out)


@pytest.mark.parametrize("dtype", DT)
def test_gelu_of_every_16_bit_value(dtype):
    """The kernels that keep the hidden layer on chip take the same GELU as the pass over memory, forward and backward, bit for bit."""
    import block_passes
    from test_gpu_mlp_backward import _backward
    x = torch.arange(-32768, 32768, device="cuda", dtype=torch.int32).to(torch.int16).view(dtype).clone()
    x[~torch.isfinite(x)] = 0
    x = x.view(256, 256)
    eye, zero, one = torch.eye(256, device="cuda", dtype=dtype), torch.zeros(256, device="cuda", dtype=dtype), torch.ones(256, D, device="cuda", dtype=dtype)
    want = block_passes.gelu(x)
    dx, _ = block_passes.gelu_backward(one, x, block_passes.scratch_for(256, 256, 256, "cuda"))
    for hidden_layer in (False, True):
        out, f = _rounded(torch.zeros_like(x), x, eye, zero, eye, zero, hidden_layer)
        assert torch.equal(out, want) and (f is None or torch.equal(f, x))      # (-0 == 0)
    _, df, g = _backward(one, x, eye, eye)
    assert torch.equal(g, want) and torch.equal(df, dx)


@pytest.mark.parametrize("dtype", DT)
@pytest.mark.parametrize("value", [float("inf"), float("-inf"), float("nan")])
def test_special_values_in_the_hidden_layer(value, dtype):
    """As in the framework: NaN for a hidden value of minus infinity, in the result and in the gradients."""
    from test_gpu_mlp_backward import _backward
    zero, eye = torch.zeros(256, D, device="cuda", dtype=dtype), torch.eye(256, device="cuda", dtype=dtype)
    b1 = zero[0].clone()
    b1[3] = value
    for hidden_layer in (False, True):
        out, f = _rounded(zero, zero, eye, b1, eye, zero[0], hidden_layer)
        want = torch.nn.functional.gelu(b1.float())
        assert torch.equal(torch.isnan(out[:, 3]), torch.isnan(want[3]).expand(256)) and (value != float("inf") or bool((out[:, 3] == value).all()))
    _, df, g = _backward(eye, b1.expand(256, 256).contiguous(), eye, eye)
    assert torch.equal(torch.isnan(g[:, 3]), torch.isnan(want[3]).expand(256)) and bool(torch.isnan(df[:, 3]).all())
    assert bool((g[:, :3] == 0).all()) and bool((g[:, 4:] == 0).all())


@pytest.mark.parametrize("B", [9, 70])      # by the passes, by the kernel
def test_a_block_gives_the_values_of_its_passes(B):
    import block_passes
    from pcf_nat_b200 import block, ops
    from pcf_nat_b200.model import NABlock
    torch.manual_seed(0)
    T, H = 150, 4
    m = torch.nn.ModuleList([NABlock(T, D, H, 7, 4, "fused")]).cuda().eval()
    with torch.no_grad():
        for n, p in m.named_parameters():      # (biases that are no 16-bit values, a hidden layer of size one)
            if "bias" in n:
                p.normal_(0, 0.3)
    blk = m[0]
    x = torch.randn(B, T, D, device="cuda").bfloat16()
    half = lambda t: t.bfloat16()
    with torch.no_grad(), torch.autocast("cuda", dtype=torch.bfloat16):
        got = block.run_blocks(m, x, None)
    with torch.no_grad():
        a = blk.attn
        linear = lambda y, lin: torch.addmm(half(lin.bias), y.view(-1, y.shape[-1]), half(lin.weight).t()).view(B, T, -1)
        h, s, _, _ = block_passes.layer_norm(x, None, blk.norm1.weight, blk.norm1.bias, blk.norm1.eps, False)
        o = ops.na1d_fused_packed(linear(h, a.qkv), H, a.win_size, a.left, 1, float(a.scale), a.relative_position_bias)
        h, s, _, _ = block_passes.layer_norm(s, linear(o, a.proj), blk.norm2.weight, blk.norm2.bias, blk.norm2.eps, False)
        want = s + linear(block_passes.gelu(linear(h, blk.fc1)), blk.fc2)
    assert float((got != want).double().mean()) <= 0.005 and float((got.double() - want.double()).norm()) <= 2e-4 * float(want.double().norm())
