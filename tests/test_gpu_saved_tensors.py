"""Saved tensors that a hook gives back as parts of larger ones, an element off their start: the nodes of blocks, layers and projections
of features give the same bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _pack(t):
    if not t.is_cuda or t.numel() == 0:
        return t
    room = torch.full((t.numel() + 8,), float("nan") if t.is_floating_point() else 0, device=t.device, dtype=t.dtype)
    return room[1:1 + t.numel()].view(t.shape).copy_(t.detach())


def _same(gradients):
    want = gradients()
    with torch.autograd.graph.saved_tensors_hooks(_pack, lambda t: t):
        got = gradients()
    assert all(torch.equal(a, b) for a, b in zip(got, want))


@pytest.mark.parametrize("layout,dim,heads,groups", [("channels_first", 64, 2, 1), ("channels_first", 64, 2, 4), ("channels_last", 256, 16, 1),
                                                     ("channels_last", 96, 2, 1)])      # (48 channels a head: split and merged)
@pytest.mark.parametrize("cast", [False, True])
def test_layer(layout, dim, heads, groups, cast):
    from pcf_nat_b200 import NAttention
    torch.manual_seed(0)
    m = NAttention(40, dim, heads, 7, 1, groups, layout=layout).cuda()
    m = m if cast else m.half()
    x = torch.randn(*((3, dim, 40) if layout == "channels_first" else (3, 40, dim)), device="cuda", dtype=torch.bfloat16 if cast else torch.float16)
    d = torch.randn_like(x)

    def gradients():
        leaf = x.clone().requires_grad_()
        with torch.autocast("cuda", dtype=torch.bfloat16, enabled=cast):
            y = m(leaf * 1)
        return torch.autograd.grad(y, [leaf] + [p for n, p in m.named_parameters() if "relative" not in n], d)

    _same(gradients)


@pytest.mark.parametrize("dim", [64, 256])
def test_blocks_and_projection(dim):
    from pcf_nat_b200 import block
    from pcf_nat_b200.model import NABlock
    torch.manual_seed(0)
    st = torch.nn.ModuleList(NABlock(40, dim, 4, 7, 4, "fused") for _ in range(2)).cuda()
    lin = torch.nn.Linear(2 * dim, dim).cuda()
    x = torch.randn(2, 40, dim, device="cuda").bfloat16()

    def gradients():
        leaf = x.clone().requires_grad_()
        with torch.autocast("cuda", dtype=torch.bfloat16):
            y = block.run_blocks(st, leaf * 1, torch.tensor([40, 31], device="cuda", dtype=torch.int32))
            z, (a, b) = block.fuse(lin, [leaf * 1, y])
        return torch.autograd.grad((z.float().sin() + a.float() + b.float().cos()).sum(),
                                   [leaf] + list(lin.parameters()) + [p for n, p in st.named_parameters() if "relative" not in n])

    _same(gradients)
