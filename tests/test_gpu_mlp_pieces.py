"""The MLP kernels (na1d_mlp_forward, na1d_mlp_backward) over many pieces of the hidden layer in a row: every second product reads
its own piece, whatever the products before and after it do."""
import pytest
import torch

pytestmark = pytest.mark.gpu
D = 256


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("rows,hidden", [(37889, 1280), (600, 1152)])
def test_every_product_reads_its_own_piece(rows, hidden, dtype):
    """Pieces of 128 whose sizes differ by powers of two up to 2^9, each read into channels of its own: a piece that is overwritten early or
    read late is off by a factor of two or more, in a few rows at least (three items and more to a pair of CTAs; 20 times)."""
    from test_gpu_mlp import _mlp
    from test_gpu_mlp_backward import _backward
    g = torch.Generator(device="cuda").manual_seed(hidden)
    rn = lambda *s: torch.randn(*s, device="cuda", generator=g)
    piece = torch.arange(hidden, device="cuda") // 128
    size = 2.0 ** (piece.float() - 4)
    into = torch.zeros(D, hidden, device="cuda")                      # channel d reads the pieces p with p = d mod 10, its own 1 of 128 columns
    for p in range(hidden // 128):
        for d in range(p, D, 10):
            into[d, 128 * p + d % 128] = 1
    h = rn(rows, D).abs().to(dtype)
    w1 = (rn(hidden, D).abs() / D * size[:, None]).to(dtype)         # (all positive: sizes of the hidden layer are those of its pieces)
    w2, zero = into.to(dtype), torch.zeros(hidden, device="cuda")
    s = torch.zeros_like(h)
    f = h.double() @ w1.double().t()
    ref = (f * torch.special.ndtr(f)) @ w2.double().t()
    u = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
    out, hid = _mlp(s, h, w1, zero, w2, torch.zeros(D, device="cuda"), True)
    assert bool(((out.double() - ref).abs() <= 4 * u * ref.abs() + 1e-4).all())      # three roundings, the first through a slope of at most 1.13
    # backward: the gradient of piece p's columns is that of its channels, times the piece's size in its own columns of w1
    x = (2 * rn(rows, hidden)).to(dtype)
    back = _backward(h, x, w1, w2)
    xd = x.double()
    slope = torch.special.ndtr(xd) + xd * torch.exp(-xd * xd / 2) * (2 * torch.pi) ** -0.5
    df = (h.double() @ w2.double()) * slope
    assert bool(((back[1].double() - df).abs() <= 2 * u * df.abs() + 1e-5).all())
    dh = back[1].double() @ w1.double()
    assert bool(((back[0].double() - dh).abs() <= 2 * u * dh.abs() + 2.0 ** -12 * (back[1].double().abs() @ w1.double().abs()) + 1e-6).all())
    for _ in range(20):
        again = _mlp(s, h, w1, zero, w2, torch.zeros(D, device="cuda"), True)
        assert torch.equal(again[0], out) and torch.equal(again[1], hid)
        assert all(torch.equal(a, b) for a, b in zip(_backward(h, x, w1, w2), back))
