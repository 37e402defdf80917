"""Parameter gradients of a layer's projections on either side of the rule that leaves large weights and bias gradients alone to the
library's products and a pass of column sums."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _gradients(m, x, d, names, hooked=False):
    handles = [lin.register_forward_hook(lambda *_: None) for lin in (m.qkv, m.proj)] if hooked else []
    params = dict(m.named_parameters())
    with torch.autocast("cuda", dtype=torch.bfloat16):
        y = m(x)
    out = torch.autograd.grad(y, [params[n] for n in names], d)
    for h in handles:
        h.remove()
    return out


# tiles of 256 x 256 of both weights: 4; 16 (four splits); 36 with few and with more rows than two splits are worth; 64 (no split), likewise
@pytest.mark.parametrize("D,heads,B,T", [(256, 4, 3, 100), (512, 8, 3, 100), (768, 12, 3, 100), (768, 12, 32, 151), (1024, 16, 3, 100), (1024, 16, 100, 201)])
@pytest.mark.parametrize("frozen", [(), ("qkv.weight",), ("qkv.weight", "proj.weight"), ("proj.weight", "proj.bias")])
def test_gradients(D, heads, B, T, frozen):
    from pcf_nat_b200 import NAttention
    torch.manual_seed(D)
    m = NAttention(T, D, heads, 7, layout="channels_last").cuda()
    x, d = (torch.randn(B, T, D, device="cuda").bfloat16() for _ in range(2))
    names = [n for n, _ in m.named_parameters() if n not in frozen and "relative" not in n]
    for n, p in m.named_parameters():
        p.requires_grad_(n not in frozen)
    for n, a, b in zip(names, _gradients(m, x, d, names), _gradients(m, x, d, names, hooked=True)):
        # module by module: three more roundings to bf16 on the way
        assert a.dtype == b.dtype and a.shape == b.shape and float((a.double() - b.double()).norm()) <= 4 * 2.0 ** -8 * float(b.double().norm()), n


def test_large_weights_need_no_room_beside_their_gradients():
    from pcf_nat_b200 import NAttention
    D = 1024
    m = NAttention(100, D, 16, 7, layout="channels_last").cuda()
    x, d = (torch.randn(2, 100, D, device="cuda").bfloat16() for _ in range(2))
    names = ["qkv.weight", "proj.weight", "qkv.bias", "proj.bias"]
    _gradients(m, x, d, names)
    params = dict(m.named_parameters())
    with torch.autocast("cuda", dtype=torch.bfloat16):
        y = m(x)
    torch.cuda.reset_peak_memory_stats()
    base = torch.cuda.memory_allocated()
    g = torch.autograd.grad(y, [params[n] for n in names], d)
    # the gradients themselves (16.8 MB) and activations of 200 rows (under 6 MB), no partial sums of the gradients' size
    assert torch.cuda.max_memory_allocated() - base <= 4 * sum(t.numel() for t in g) + 8 * 2 ** 20
