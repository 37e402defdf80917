"""Parameter gradients of projections in one launch (na1d_projection_gradients) against the same products in 64 bits."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


def _gradients(pairs, out32, weights=True, biases=True):
    from pcf_nat_b200 import _lib
    L, n, rows = _lib.lib(), len(pairs), pairs[0][0].shape[0]
    M, N = ((ctypes.c_int64 * n)(*[t[i].shape[1] for t in pairs]) for i in (0, 1))
    scratch = torch.full((L.na1d_projection_gradients_scratch(M, N, n, rows),), float("nan"), device="cuda")
    dt = torch.float32 if out32 else pairs[0][0].dtype
    # a guard of 64 elements behind every result
    w = [torch.full((a.shape[1] * b.shape[1] + 64,), 7.0, device="cuda", dtype=dt) for a, b in pairs]
    c = [torch.full((a.shape[1] + 64,), 7.0, device="cuda", dtype=dt) for a, b in pairs]
    pointers = lambda ts, on=True: (ctypes.c_void_p * n)(*[t.data_ptr() if on else None for t in ts])
    _lib.check(L.na1d_projection_gradients(pointers(w, weights), pointers(c, biases), pointers([a for a, _ in pairs]), pointers([b for _, b in pairs]), M, N, n,
                                           rows, scratch.data_ptr(), int(out32), _lib.NA1D_BF16 if pairs[0][0].dtype == torch.bfloat16 else _lib.NA1D_FP16,
                                           torch.cuda.current_stream().cuda_stream), "na1d_projection_gradients")
    assert L.na1d_device_status() == 0
    for t in w + c:
        assert bool((t[-64:] == 7.0).all())
    return [t[:-64].view(a.shape[1], b.shape[1]) for t, (a, b) in zip(w, pairs)], [t[:-64] for t in c]


# tiles of 256 x 256, steps of 64 rows, at least four steps to a split: sizes on and beside each edge, one round of CTA pairs and more
@pytest.mark.parametrize("rows,shapes", [
    (1, [(8, 8)]), (63, [(64, 256), (8, 264)]), (64, [(256, 256)]), (65, [(264, 8), (248, 520)]), (257, [(768, 256), (256, 256)]),
    (1000, [(384, 128), (128, 128)]), (5003, [(1536, 512), (512, 512)]), (300, [(2560, 2048), (256, 8)]), (38400, [(1024, 256), (256, 1024)])])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_parameter_gradients(rows, shapes, dtype):
    g = torch.Generator(device="cuda").manual_seed(rows)
    pairs = [tuple(torch.randn(rows, k, device="cuda", generator=g).to(dtype) for k in s) for s in shapes]
    w, b = _gradients(pairs, True)
    w16, b16 = _gradients(pairs, False)
    for i, (dy, x) in enumerate(pairs):
        rw, rb = dy.double().t() @ x.double(), dy.double().sum(0)
        # exact products, fp32 sums of `rows` terms of size one: each addition rounds a partial sum of at most the square root of the
        # number of terms by 2^-23 of itself (towards zero at worst), so rows * 2^-23 * sqrt(rows) bounds the largest error
        bound = rows * 2.0 ** -23 * rows ** 0.5 * 4
        assert float((w[i].double() - rw).abs().max()) <= bound
        assert float((b[i].double() - rb).abs().max()) <= bound
        # 16-bit results are the fp32 ones rounded once
        assert torch.equal(w16[i], w[i].to(dtype)) and torch.equal(b16[i], b[i].to(dtype))
    again = _gradients(pairs, True)
    assert all(torch.equal(p, q) for p, q in zip(w + b, again[0] + again[1]))


def test_parameter_gradients_one_kind_alone():
    g = torch.Generator(device="cuda").manual_seed(3)
    pairs = [tuple(torch.randn(700, k, device="cuda", generator=g).bfloat16() for k in (768, 256))]
    w, b = _gradients(pairs, True)
    assert torch.equal(_gradients(pairs, True, biases=False)[0][0], w[0])
    assert torch.equal(_gradients(pairs, True, weights=False)[1][0], b[0])
    assert bool((_gradients(pairs, True, weights=False)[0][0] == 7.0).all())


def test_layer_input_off_a_16_byte_boundary():
    from pcf_nat_b200 import NAttention
    torch.manual_seed(0)
    m = NAttention(40, 64, 4, 7, layout="channels_last").cuda().half()
    x = torch.randn(2 * 40 * 64 + 1, device="cuda").half()
    d = torch.randn(2, 40, 64, device="cuda").half()
    out = []
    for t in (x[1:].view(2, 40, 64), x[1:].clone().view(2, 40, 64)):
        t = t.detach().requires_grad_(True)
        out.append(torch.autograd.grad(m(t), [t] + list(m.parameters()), d))
    assert all(torch.equal(p, q) for p, q in zip(*out))
