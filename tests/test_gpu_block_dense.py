"""Blocks of shapes that the kernels on the packed projection do not take: one node around the dense operator, against the modules."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _blocks(dim, heads, T, win, n=2):
    from pcf_nat_b200.model import NABlock
    torch.manual_seed(dim + win)
    st = torch.nn.ModuleList(NABlock(T, dim, heads, win, 4, "fused") for _ in range(n)).cuda()
    for b in st:
        torch.nn.init.normal_(b.attn.relative_position_bias, std=0.3)
    return st


def _run(st, x, dtype, node, padding=None):
    from pcf_nat_b200 import block
    with torch.autocast("cuda", dtype=dtype):
        if node:
            y = block.run_blocks(st, x, None if padding is None else x.shape[1] - padding)
            assert y is not None
            return y
        for b in st:
            x = b(x, padding)
        return x


# 64 channels a head at a window without room for the bias gradient, head sizes outside the packed ones, one token, the widest window
@pytest.mark.parametrize("dim,heads,T,win", [(256, 4, 131, 27), (256, 4, 40, 33), (96, 2, 77, 15), (192, 2, 65, 41), (128, 1, 1, 7), (48, 2, 150, 80)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_gradients(dim, heads, T, win, dtype):
    from pcf_nat_b200 import ops
    assert not ops.packed_supported(heads, T, dim // heads, win, win // 2, 1, dtype)
    st = _blocks(dim, heads, T, win)
    st[0].attn.qkv.weight.requires_grad_(False)
    st[1].attn.relative_position_bias.requires_grad_(False)
    x = torch.randn(3, T, dim, device="cuda").to(dtype).requires_grad_()
    leaves = [x] + [p for p in st.parameters() if p.requires_grad]
    got, want = ([y] + list(torch.autograd.grad(y.float().sin().sum(), leaves)) for y in (_run(st, x, dtype, True), _run(st, x, dtype, False)))
    # about eight 16-bit tensors deep in either way
    u = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
    for i, (a, b) in enumerate(zip(got, want)):
        assert a.dtype == b.dtype and a.shape == b.shape
        assert float((a.double() - b.double()).norm()) <= 8 * u * float(b.double().norm()) + 1e-4, i


@pytest.mark.parametrize("dim,heads,T,win", [(256, 4, 131, 27), (96, 2, 77, 15)])
def test_evaluation_with_padding(dim, heads, T, win):
    st = _blocks(dim, heads, T, win).eval()
    x = torch.randn(3, T, dim, device="cuda").to(torch.bfloat16)
    padding = torch.tensor([0, 5, T - 1], device="cuda")
    with torch.no_grad():
        a, b = _run(st, x, torch.bfloat16, True, padding), _run(st, x, torch.bfloat16, False, padding)
    assert float((a.double() - b.double()).norm()) <= 8 * 2.0 ** -8 * float(b.double().norm())


def test_second_derivative():
    st = _blocks(256, 4, 40, 33)
    got = []
    for node in (True, False):
        x = torch.randn(2, 40, 256, device="cuda", generator=torch.Generator(device="cuda").manual_seed(1)).to(torch.bfloat16).requires_grad_()
        y = _run(st, x, torch.bfloat16, node)
        g, = torch.autograd.grad(y.float().pow(2).sum(), x, create_graph=True)
        leaves = [x] + list(st.parameters())
        out = torch.autograd.grad(g.float().pow(2).sum(), leaves, allow_unused=True)
        got.append([g.detach()] + [torch.zeros_like(p) if o is None else o for o, p in zip(out, leaves)])
    for a, b in zip(*got):
        assert float((a.double() - b.double()).norm()) <= 8 * 2.0 ** -8 * float(b.double().norm()) + 1e-4
