"""A projection of tensors side by side as one node (block.fuse) against the concatenation and the layer."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _run(kind, lin, xs, stages, dtype, order):
    """A chain as in the network: each stage projects all features so far; what comes out is a feature too. Loss over all of them side by
    side (slices of a wide gradient), `order` 2: a gradient penalty."""
    from pcf_nat_b200 import block
    with torch.autocast("cuda", dtype=dtype):
        feats, x = [xs[0] * 1], None
        for s in range(stages):
            feats.append(xs[s + 1] * 1 if x is None else torch.tanh(x) + xs[s + 1])
            got = block.fuse(lin[s], feats) if kind == "node" else None
            assert (got is None) == (kind != "node")
            x, feats = (lin[s](torch.cat(feats, -1)), feats) if got is None else got
        wide = torch.cat(feats[1:] + [x], -1).float()
    loss = (wide * torch.linspace(-1, 1, wide.shape[-1], device="cuda")).sin().sum()
    leaves = [t for t in list(xs[:stages + 1]) + [p for l in lin for p in l.parameters()] if t.requires_grad]
    if order == 1:
        return [wide.detach()] + list(torch.autograd.grad(loss, leaves))
    g, = torch.autograd.grad(loss, xs[0], create_graph=True)
    second = torch.autograd.grad(g.float().pow(2).sum(), leaves, allow_unused=True)
    return [g.detach()] + [torch.zeros_like(t) if o is None else o for t, o in zip(leaves, second)]


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("N,T,D,stages,order", [(1, 1, 8, 1, 1), (2, 50, 64, 3, 1), (3, 33, 40, 2, 1), (8, 300, 256, 5, 1), (2, 50, 64, 3, 2)])
@pytest.mark.parametrize("frozen", [False, True])
def test_fuse(N, T, D, stages, order, dtype, frozen):
    torch.manual_seed(N * T + D)
    lin = [torch.nn.Linear((s + 2) * D, D).cuda() for s in range(stages)]
    xs = [torch.randn(N, T, D, device="cuda").to(dtype).requires_grad_() for _ in range(stages + 1)]
    if frozen:
        lin[0].weight.requires_grad_(False)
        lin[-1].bias.requires_grad_(False)
        xs[-1].requires_grad_(False)
    node, ops = (_run(kind, lin, xs, stages, dtype, order) for kind in ("node", "operations"))
    # the chain is about four 16-bit tensors to a stage deep, in both; sums here are rounded once, there at every step
    u = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
    for i, (a, b) in enumerate(zip(node, ops)):
        assert a.dtype == b.dtype and a.shape == b.shape
        assert float((a.double() - b.double()).norm()) <= 4 * (stages + 1) * u * float(b.double().norm()) + 1e-5, i
    assert len(node) == len(ops)
    if order == 1 and dtype == torch.bfloat16 and not frozen:   # no further off than the operations
        ref = _exact(lin, xs, stages)
        for a, b, r in zip(node[1:], ops[1:], ref):
            assert float((a.double() - r).norm()) <= 1.1 * float((b.double() - r).norm()) + 1e-5


def _exact(lin, xs, stages):
    ys = [t.detach().double().requires_grad_() for t in xs]
    ps = [[p.detach().double().requires_grad_() for p in l.parameters()] for l in lin]
    feats, x = [ys[0]], None
    for s in range(stages):
        feats.append(ys[s + 1] if x is None else torch.tanh(x) + ys[s + 1])
        x = torch.cat(feats, -1) @ ps[s][0].t() + ps[s][1]
    wide = torch.cat(feats[1:] + [x], -1)
    loss = (wide * torch.linspace(-1, 1, wide.shape[-1], device="cuda")).sin().sum()
    return torch.autograd.grad(loss, ys + [p for l in ps for p in l])


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_one_part_that_is_read_again(dtype):
    """As in the pooling: a projection of one tensor, which what follows reads too."""
    from pcf_nat_b200 import block
    torch.manual_seed(0)
    lin = torch.nn.Linear(384, 128).cuda()
    x = torch.randn(3, 41, 384, device="cuda").to(dtype).requires_grad_()
    out = []
    for node in (True, False):
        with torch.autocast("cuda", dtype=dtype):
            y, again = block.fuse(lin, [x]) if node else (lin(x), [x])
        assert y.dtype == dtype and torch.equal(again[0], x)
        loss = (y.float().sin().sum(-1, keepdim=True) * again[0].float().cos()).sum()
        out.append([y.detach()] + list(torch.autograd.grad(loss, [x] + list(lin.parameters()))))
    u = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
    for a, b in zip(*out):
        assert a.dtype == b.dtype and float((a.double() - b.double()).norm()) <= 4 * u * float(b.double().norm()) + 1e-5


def test_left_to_the_operations():
    from pcf_nat_b200 import block
    lin = torch.nn.Linear(128, 64).cuda()
    x = torch.randn(2, 9, 64, device="cuda", dtype=torch.bfloat16)
    with torch.autocast("cuda", dtype=torch.bfloat16):
        assert block.fuse(lin, [x, x]) is not None
        assert block.fuse(lin, [x, x.transpose(0, 1).contiguous().transpose(0, 1)]) is None and block.fuse(lin, [x, x.half()]) is None
        assert block.fuse(lin, [x, x, x]) is None and block.fuse(torch.nn.Linear(128, 64, bias=False).cuda(), [x, x]) is None
        assert block.fuse(lin.cuda().double(), [x, x]) is None
        lin.float()
        with torch.no_grad():
            assert block.fuse(lin, [x, x]) is None
        handle = lin.register_forward_hook(lambda *a: None)
        assert block.fuse(lin, [x, x]) is None
        handle.remove()
    assert block.fuse(lin, [x, x]) is None      # without autocast
    with torch.autocast("cuda", dtype=torch.float16):
        assert block.fuse(lin, [x, x]) is None


@pytest.mark.parametrize("D", [64, 256])
def test_saved_tensors_may_come_back_inside_others(D):
    """What the nodes save may be given back as parts of larger tensors, 16 bytes off their start: the gradients stay the same bits."""
    from pcf_nat_b200 import block
    from pcf_nat_b200.model import NABlock
    torch.manual_seed(0)
    st = torch.nn.ModuleList(NABlock(40, D, 4, 7, 4, "fused") for _ in range(2)).cuda()
    lin = torch.nn.Linear(2 * D, D).cuda()
    x = torch.randn(2, 40, D, device="cuda").to(torch.bfloat16).requires_grad_()

    def pack(t):
        if not t.is_cuda or t.numel() == 0:
            return t
        room = torch.full((t.numel() + 64,), float("nan") if t.is_floating_point() else 0, device=t.device, dtype=t.dtype)
        return room[8:8 + t.numel()].view(t.shape).copy_(t.detach())

    def gradients():
        with torch.autocast("cuda", dtype=torch.bfloat16):
            y = block.run_blocks(st, x, None)
            z, (a, b) = block.fuse(lin, [x, y])
        return torch.autograd.grad((z.float().sin() + a.float() + b.float().cos()).sum(),
                                   [x] + list(lin.parameters()) + [p for n, p in st.named_parameters() if "relative" not in n])

    want = gradients()
    with torch.autograd.graph.saved_tensors_hooks(pack, lambda t: t):
        got = gradients()
    for a, b in zip(got, want):
        assert torch.equal(a, b)
