"""The C++ autograd nodes against the Python ones: the same bits, the same saved-tensor and error behaviour, and the calls they
leave to the Python route."""
import threading

import pytest
import torch

pytestmark = pytest.mark.gpu


def _args(T=70, C=32, dtype=torch.bfloat16, bias_dtype=torch.float32, heads=2, batch=3, win=7):
    g = torch.Generator(device="cuda").manual_seed(1)
    q, k, v = (torch.randn(batch * heads, T, C, device="cuda", generator=g).to(dtype).requires_grad_() for _ in range(3))
    rpb = torch.randn(1, heads, 1, win, device="cuda", generator=g).to(bias_dtype).requires_grad_()
    d_o = torch.randn(batch * heads, T, C, device="cuda", generator=g).to(dtype)
    return q, k, v, rpb, d_o


def _python(q, k, v, rpb, vl, heads, drop=0.0):
    from pcf_nat_b200 import NA1dFusedFunction
    return NA1dFusedFunction.apply(q, k, v, 7, 3, 1, 0.2, rpb, vl, heads, drop, 5)


@pytest.mark.parametrize("C,drop,padded,bias_dtype", [(32, 0.0, False, torch.float32), (32, 0.1, True, torch.float32), (48, 0.0, True, torch.bfloat16),
                                                      (16, 0.0, True, None)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_operator_node_gives_the_python_nodes_bits(C, drop, padded, bias_dtype, dtype):
    from pcf_nat_b200 import na1d_fused, ops
    q, k, v, rpb, d_o = _args(C=C, dtype=dtype, bias_dtype=bias_dtype or torch.float32)
    rpb = rpb if bias_dtype else None
    vl = torch.tensor([70, 31, 0], device="cuda") if padded else None
    o = na1d_fused(q, k, v, 7, 3, 1, 0.2, rpb, vl, 2, drop, 5)
    p = _python(q, k, v, rpb, vl, 2, drop)
    assert o.grad_fn.name() != p.grad_fn.name()
    assert torch.equal(o, p)
    leaves = [q, k, v] + ([rpb] if rpb is not None else [])
    a, b = torch.autograd.grad(o, leaves, d_o, retain_graph=True), torch.autograd.grad(p, leaves, d_o)
    for x, y in zip(a[:3], b[:3]):
        assert torch.equal(x, y)
    for x, y in zip(a[3:], b[3:]):      # atomics: the order of the CTAs' sums
        assert x.shape == y.shape and x.dtype == y.dtype and torch.allclose(x, y, rtol=1e-2 if x.dtype != torch.float32 else 1e-4, atol=1e-4)
    again = torch.autograd.grad(o, q, d_o)[0]      # a second pass over the kept graph, for one input only
    assert torch.equal(again, a[0])
    with torch.no_grad():
        assert torch.equal(na1d_fused(q, k, v, 7, 3, 1, 0.2, rpb, vl, 2, drop, 5), o)
    if padded:
        assert torch.equal(na1d_fused(q, k, v, 7, 3, 1, 0.2, rpb, vl.cpu(), 2, drop, 5), o)
        assert torch.equal(na1d_fused(q, k, v, 7, 3, 1, 0.2, rpb, vl.tolist(), 2, drop, 5), o)
    ops.device_status()


def test_packed_node_gives_the_python_nodes_bits():
    from pcf_nat_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(2)
    qkv = torch.randn(3, 70, 3 * 64, device="cuda", generator=g).bfloat16().requires_grad_()
    rpb = torch.randn(1, 2, 1, 9, device="cuda", generator=g).requires_grad_()
    vl = torch.tensor([70, 12, 44], device="cuda", dtype=torch.int32)
    d = torch.randn(3, 70, 64, device="cuda", generator=g).bfloat16()
    o = ops.na1d_fused_packed(qkv, 2, 9, 4, 3, 0.2, rpb, vl)
    p = ops.NA1dFusedPackedFunction.apply(qkv, 2, 9, 4, 3, 0.2, rpb, vl)
    assert torch.equal(o, p) and o.grad_fn.name() != p.grad_fn.name()
    a, b = torch.autograd.grad(o, (qkv, rpb), d), torch.autograd.grad(p, (qkv, rpb), d)
    assert torch.equal(a[0], b[0]) and torch.allclose(a[1], b[1], rtol=1e-4, atol=1e-4)
    rpb.requires_grad_(False)
    o = ops.na1d_fused_packed(qkv, 2, 9, 4, 3, 0.2, rpb, vl)
    assert torch.equal(torch.autograd.grad(o, qkv, d)[0], a[0])


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_pair_nodes_give_the_python_nodes_bits(dtype):
    from pcf_nat_b200 import getNA1dFunction
    q, k, v, _, d_o = _args(dtype=dtype)
    out = []
    for call in (lambda f, *a: f.apply(*a), lambda f, *a: super(f, f).apply(*a)):     # the C++ node, the class itself
        QK, AV = getNA1dFunction(32, 1, dtype)
        attn = call(QK, q, k, 7, 3, 1)
        o = call(AV, attn.softmax(-1), v, 7, 3, 1)
        out.append([attn, o] + list(torch.autograd.grad(o, (q, k, v), d_o)))
    for a, b in zip(*out):
        assert a.dtype == b.dtype and torch.equal(a, b)
    assert out[0][0].grad_fn.name() != out[1][0].grad_fn.name()
    other = torch.float16 if dtype == torch.bfloat16 else torch.bfloat16
    with pytest.raises(AssertionError):
        getNA1dFunction(32, 1, other)[0].apply(q, k, 7, 3, 1)
    with pytest.raises(AssertionError):
        QK.apply(q.transpose(0, 1), k.transpose(0, 1), 7, 3)
    with torch.no_grad():
        assert torch.equal(QK.apply(q, k, 7, 3), out[0][0])


def test_saved_tensor_hooks_see_what_is_saved():
    from pcf_nat_b200 import na1d_fused
    q, k, v, rpb, d_o = _args()
    seen = []

    def pack(t):
        seen.append(t)
        return t.cpu()

    want = torch.autograd.grad(na1d_fused(q, k, v, 7, 3, 1, 0.2, rpb, None, 2), q, d_o)[0]
    with torch.autograd.graph.saved_tensors_hooks(pack, lambda t: t.cuda()):
        o = na1d_fused(q, k, v, 7, 3, 1, 0.2, rpb, None, 2)
    assert len(seen) >= 5
    assert torch.equal(torch.autograd.grad(o, q, d_o)[0], want)


def test_errors_are_the_packages_own():
    from pcf_nat_b200 import na1d_fused
    from pcf_nat_b200._lib import Na1dError
    q, k, v, rpb, d_o = _args()
    with pytest.raises(Na1dError) as e:
        na1d_fused(q, k, v, 7, 7, 1, 0.2, None, None, 2)
    assert e.value.status == -3
    with pytest.raises(Na1dError):
        na1d_fused(q, k, v, 7, 3, 1, 0.2, None, None, 4)               # N not a multiple of heads
    with pytest.raises(AssertionError):
        na1d_fused(q.transpose(1, 2), k, v, 7, 3)
    with pytest.raises(Exception):
        na1d_fused(q, k, v.half(), 7, 3)
    with pytest.raises(RuntimeError, match="CUDA"):
        na1d_fused(q.cpu(), k.cpu(), v.cpu(), 7, 3)
    # an error inside the backward reaches the caller as the same class: a bias gradient table above its capacity
    q, k, v, rpb, d_o = _args(heads=150, batch=1, win=100)
    o = na1d_fused(q, k, v, 100, 50, 1, 0.2, rpb, None, 150)
    with pytest.raises(Na1dError) as e:
        torch.autograd.grad(o, rpb, d_o)
    assert e.value.status == -9
    q2 = q.detach().requires_grad_()
    o = na1d_fused(q2, k, v, 100, 50, 1, 0.2, rpb, None, 150)
    q2.data.mul_(1)
    with torch.no_grad():
        q2.mul_(2)                                                      # saved tensors are version-checked
    with pytest.raises(RuntimeError, match="inplace|in-place|modified"):
        torch.autograd.grad(o, k, d_o)


def test_transforms_take_the_python_route():
    from pcf_nat_b200 import na1d_fused
    q, k, v, rpb, d_o = (t.detach() for t in _args())
    with pytest.raises(RuntimeError):
        torch.func.vmap(lambda a: na1d_fused(a, k, v, 7, 3))(torch.stack([q, q]))
    with pytest.raises(RuntimeError):
        torch.func.grad(lambda a: na1d_fused(a, k, v, 7, 3).float().sum())(q)
    with torch.autograd.forward_ad.dual_level(), pytest.raises(Exception):
        torch.autograd.forward_ad.unpack_dual(na1d_fused(torch.autograd.forward_ad.make_dual(q, q), k, v, 7, 3))


def test_streams_and_threads():
    """Concurrent calls from several threads on streams of their own give what one call gives."""
    from pcf_nat_b200 import na1d_fused
    q, k, v, rpb, d_o = _args(T=300)
    want = torch.autograd.grad(na1d_fused(q, k, v, 7, 3, 1, 0.2, rpb, None, 2), q, d_o)[0]
    torch.cuda.synchronize()
    got = [None] * 4

    def work(i):
        s = torch.cuda.Stream()
        with torch.cuda.stream(s):
            for _ in range(20):
                a = q.detach().requires_grad_()
                got[i] = torch.autograd.grad(na1d_fused(a, k, v, 7, 3, 1, 0.2, rpb, None, 2), a, d_o)[0]
        s.synchronize()

    ts = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert all(torch.equal(g, want) for g in got)


def test_valid_tokens():
    from pcf_nat_b200.nattention import _valid_tokens
    for pad in (torch.tensor([0, 5, 100, -3]), torch.tensor([7]), torch.tensor([2, 0, 1, 9], dtype=torch.int32), torch.tensor(4), torch.tensor([1.0, 2.0, 0.0, 60.0])):
        want = (50 - pad.to(torch.int64)).clamp_(0, 50).to(torch.int32).expand(4)
        got = _valid_tokens(50, pad.cuda(), 4)
        assert got.dtype == torch.int32 and got.is_contiguous() and torch.equal(got.cpu(), want)


def test_subclasses_of_the_pair_run_their_own_forward():
    from pcf_nat_b200 import getNA1dFunction
    q, k, v, _, _ = _args()
    QK, AV = getNA1dFunction(32, 1, torch.bfloat16)

    class Twice(QK):
        @staticmethod
        def forward(ctx, *a):
            return 2 * QK.forward(ctx, *a)

    class TwiceAV(AV):
        @staticmethod
        def forward(ctx, *a):
            return 2 * AV.forward(ctx, *a)

    attn = QK.apply(q, k, 7, 3)
    assert torch.equal(Twice.apply(q, k, 7, 3), 2 * attn)
    assert torch.equal(TwiceAV.apply(attn, v, 7, 3), 2 * AV.apply(attn, v, 7, 3))


def test_every_route_without_the_extension():
    """The operator, the pair, both layers and the network on the Python routes alone, in a process that cannot import the nodes."""
    import os
    import subprocess
    import sys

    from test_block_routes_cpu import WITHOUT_NODES
    program = WITHOUT_NODES + """
import torch
from pcf_nat_b200.model import PCFNATExtractor
g = lambda *s: torch.randn(*s, device="cuda").half().requires_grad_()
q, k, v = g(4, 50, 32), g(4, 50, 32), g(4, 50, 32)
QK, AV = pcf_nat_b200.getNA1dFunction(32, 1, torch.float16)
a = AV.apply(QK.apply(q, k, 7, 3).softmax(-1), v, 7, 3)
o = pcf_nat_b200.na1d_fused(q, k, v, 7, 3)
assert "Backward" in o.grad_fn.name() and torch.allclose(a[:, 3:-3], o[:, 3:-3], atol=1e-2)     # (no mask at the ends)
torch.autograd.grad(o.float().sum() + a.float().sum(), (q, k, v))
for layout in ("channels_first", "channels_last"):
    m = pcf_nat_b200.NAttention(50, 64, 2, 7, layout=layout).cuda().half()
    x = g(2, 64, 50) if layout == "channels_first" else g(2, 50, 64)
    m(x).float().sum().backward()
    with torch.no_grad():
        m.eval()(x, torch.tensor([0, 9], device="cuda"))
m = PCFNATExtractor(frames=40, feat=16, dim=32, heads=2, win=5, stages=2, blocks=1, emb=16, classes=10).cuda()
with torch.autocast("cuda", dtype=torch.bfloat16):
    m(torch.randn(4, 16, 40, device="cuda"), torch.arange(4, device="cuda")).backward()
    with torch.no_grad():
        m.eval().embedding(torch.randn(4, 16, 40, device="cuda"), torch.tensor([0, 1, 2, 3]))
torch.cuda.synchronize()
"""
    subprocess.run([sys.executable, "-c", program], cwd=os.path.dirname(os.path.dirname(os.path.abspath(__file__))), check=True)
