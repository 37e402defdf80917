"""The general kernels on warp-level matrix instructions against plain PyTorch in 64 bits and against the CUDA-core kernels:
every padded channel count, windows around a multiple of the 16-row chunk, asymmetric and one-sided windows, dilations with
empty and uneven residues, sequences shorter than a tile and around its 64 rows, padding, values that are not finite."""
import pytest
import torch

pytestmark = pytest.mark.gpu

#      B  H  T    C   win left dil bias  padded
CASES = [
    (1, 1, 1, 8, 1, 0, 1, True, False),
    (2, 3, 64, 8, 80, 40, 1, True, True),
    (1, 2, 65, 16, 34, 33, 1, False, True),
    (2, 4, 203, 48, 41, 20, 1, True, True),
    (1, 2, 130, 24, 7, 0, 3, True, False),
    (2, 1, 5, 48, 9, 4, 7, True, True),          # more residues than tokens
    (1, 2, 63, 96, 17, 8, 2, True, True),
    (1, 2, 150, 128, 33, 16, 1, False, False),
    (1, 1, 200, 128, 128, 64, 1, True, True),
    (1, 2, 97, 64, 50, 3, 1, True, True),
    (1, 1, 300, 32, 49, 48, 4, True, False),
    (1, 40, 50, 16, 18, 9, 1, True, True),        # more heads than the tcgen05 kernels take
]


def _inputs(case, dtype, seed=0):
    B, H, T, C, win, left, dil, bias, padded = case
    g = torch.Generator(device="cuda").manual_seed(seed)
    q, k, v, d_o = (torch.randn(B * H, T, C, device="cuda", generator=g).to(dtype) for _ in range(4))
    rpb = torch.randn(H, win, device="cuda", generator=g) if bias else None
    vl = torch.randint(0, T + 1, (B,), device="cuda", generator=g, dtype=torch.int32) if padded else None
    return q, k, v, d_o, rpb, vl


def _reference(case, q, k, v, d_o, rpb, vl):
    B, H, T, C, win, left, dil, _, _ = case
    q, k, v = (x.double().view(B, H, T, C).requires_grad_() for x in (q, k, v))
    r = None if rpb is None else rpb.double().requires_grad_()
    j = torch.arange(T, device="cuda")[:, None] + (torch.arange(win, device="cuda") - left) * dil
    inr = (j >= 0) & (j < T)
    n = torch.full((B, 1, 1), T, device="cuda") if vl is None else vl.view(B, 1, 1)
    masked = (j < 0) | (j >= n) | (torch.arange(T, device="cuda").view(1, T, 1) >= n)
    kg, vg = (x[:, :, j.clamp(0, T - 1)] * inr[..., None] for x in (k, v))
    x = torch.einsum("bhtc,bhtwc->bhtw", q, kg) * C ** -0.5 - 100.0 * masked[:, None]
    p = torch.softmax(x if r is None else x + r[None, :, None], -1)
    o = torch.einsum("bhtw,bhtwc->bhtc", p, vg)
    grads = torch.autograd.grad(o, [q, k, v] + ([] if r is None else [r]), d_o.double().view(B, H, T, C))
    return [t.detach().reshape(B * H, T, C) for t in (o,) + grads[:3]] + list(grads[3:])


def _run(family, case, q, k, v, d_o, rpb, vl):
    from pcf_nat_b200 import ops
    B, H, T, C, win, left, dil, _, _ = case
    old = ops.set_kernel_family(family)
    try:
        o, lse = ops.fused_forward(q, k, v, win, left, dil, C ** -0.5, rpb, vl, H)
        dq, dk, dv, dr = ops.fused_backward(d_o, q, k, v, o, lse, win, left, dil, C ** -0.5, rpb, vl, H, need_d_rpb=rpb is not None)
    finally:
        ops.set_kernel_family(old)
    return [o, dq, dk, dv] + ([] if dr is None else [dr])


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("case", CASES)
def test_against_64_bits_and_the_cuda_core_kernels(case, dtype):
    from pcf_nat_b200 import ops
    args = _inputs(case, dtype)
    ref = _reference(case, *args)
    mma, core = _run(ops.FAMILY_WARP_MMA, case, *args), _run(ops.FAMILY_CUDA_CORE, case, *args)
    eps = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
    for i, (a, b, r) in enumerate(zip(mma, core, ref)):
        ea, eb, n = float((a.double() - r).norm()), float((b.double() - r).norm()), float(r.norm())
        # both are one 16-bit rounding of an fp32 result: their errors agree but for the scatter of a few elements that round the
        # other way (the fp32 bias gradient: its own summation order)
        assert ea <= eb * (1.02 + 2 / r.numel() ** 0.5) + (1e-6 if i < 4 else 4e-6) * n + 1e-6, (i, ea, eb, n)
        # delta uses the rounded output, as the CUDA-core kernel does: its rounding enters the gradients
        assert float((a.double() - r).abs().max()) <= 4 * eps * float(r.abs().max()) + 1e-5, i


@pytest.mark.parametrize("scale", [1e-4, 3e3])
def test_gradients_far_from_one_keep_their_precision(scale):
    """fp16 output gradients near both ends of their range: dS must not lose bits to an fp16 exponent on the way."""
    from pcf_nat_b200 import ops
    case = (1, 2, 100, 48, 41, 20, 1, True, False)
    q, k, v, d_o, rpb, vl = _inputs(case, torch.float16)
    args = (q, k, v, (d_o.float() * scale).to(torch.float16), rpb, vl)
    ref = _reference(case, *args)
    for a, b, r in zip(_run(ops.FAMILY_WARP_MMA, case, *args), _run(ops.FAMILY_CUDA_CORE, case, *args), ref):
        ok = torch.isfinite(b.double())
        assert torch.equal(ok, torch.isfinite(a.double()))
        ea, eb = float((a.double() - r)[ok].norm()), float((b.double() - r)[ok].norm())
        assert ea <= 1.05 * eb + 4e-6 * float(r.norm()), (ea, eb)


@pytest.mark.parametrize("which", [0, 1, 2, 3])
@pytest.mark.parametrize("value", [float("nan"), float("inf")])
def test_values_that_are_not_finite_reach_their_window_only(which, value):
    from pcf_nat_b200 import ops
    case = (1, 1, 150, 48, 9, 4, 1, True, False)
    args = _inputs(case, torch.bfloat16)
    args[which][0, 70, 5] = value
    for i, (a, r) in enumerate(zip(_run(ops.FAMILY_WARP_MMA, case, *args), _reference(case, *args))):
        ok = torch.isfinite(r)
        assert torch.equal(ok, torch.isfinite(a)), (i, int((~ok).sum()), int((~torch.isfinite(a)).sum()))
        if bool(ok.any()):
            assert float((a.double() - r)[ok].abs().max()) <= 2.0 ** -6 * float(r[ok].abs().max()), i


def test_routes():
    """Above 128 channels and for few neighbours the CUDA-core kernels stay; the automatic route of a general shape is the warp-level
    one, bit for bit."""
    from pcf_nat_b200 import ops
    case = (64, 4, 20, 8, 5, 2, 4, True, True)
    args = _inputs(case, torch.bfloat16)
    for a, b in zip(_run(ops.FAMILY_AUTO, case, *args)[:4], _run(ops.FAMILY_CUDA_CORE, case, *args)[:4]):
        assert torch.equal(a, b)
    case = (16, 8, 300, 48, 20, 9, 1, True, True)
    args = _inputs(case, torch.bfloat16)
    for a, b in zip(_run(ops.FAMILY_AUTO, case, *args)[:4], _run(ops.FAMILY_WARP_MMA, case, *args)[:4]):
        assert torch.equal(a, b)
    case = (1, 2, 70, 192, 20, 9, 1, True, True)
    args = _inputs(case, torch.bfloat16)
    for a, b in zip(_run(ops.FAMILY_WARP_MMA, case, *args)[:4], _run(ops.FAMILY_CUDA_CORE, case, *args)[:4]):
        assert torch.equal(a, b)


def _pair_reference(q, k, attn, win, left, dil):
    """(q.k over the window, attn . k, transposed attn . q) in 64 bits; rows outside the sequence are zero rows."""
    N, T, C = q.shape
    j = torch.arange(T, device="cuda")[:, None] + (torch.arange(win, device="cuda") - left) * dil
    inr = ((j >= 0) & (j < T)).double()
    jc = j.clamp(0, T - 1)
    kg = k.double()[:, jc] * inr[None, :, :, None]
    a = attn.double() * inr
    out = torch.zeros(N, T, C, device="cuda", dtype=torch.float64)
    out.index_add_(1, jc.reshape(-1), (a[..., None] * q.double()[:, :, None]).reshape(N, T * win, C))
    return torch.einsum("ntc,ntwc->ntw", q.double(), kg), torch.einsum("ntw,ntwc->ntc", a, kg), out


@pytest.mark.parametrize("family", [-1, 0, 3, 4])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("N,T,C,win,left,dil", [(1, 1, 8, 1, 0, 1), (3, 128, 16, 27, 13, 1), (2, 129, 16, 5, 0, 1), (2, 150, 32, 33, 32, 1), (3, 97, 48, 41, 20, 1),
                                                (2, 300, 64, 9, 4, 1), (2, 300, 64, 18, 4, 3), (1, 260, 128, 128, 64, 1), (2, 7, 24, 9, 4, 5),
                                                (2, 40, 192, 12, 3, 1), (1, 1, 16, 33, 0, 1), (5, 31, 16, 17, 16, 1), (2, 1500, 16, 18, 2, 1),
                                                (700, 150, 16, 1, 0, 1)])
def test_unfused_operators(N, T, C, win, left, dil, dtype, family):
    """All routes of the six unfused entry points: fp32 results to fp32 accuracy (the band in), 16-bit results to their rounding --
    half a step, plus the tcgen05 kernels' 16-bit band, at most another half step per term."""
    from pcf_nat_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(4)
    q, k = (torch.randn(N, T, C, device="cuda", generator=g).to(dtype) for _ in range(2))
    attn = torch.randn(N, T, win, device="cuda", generator=g)
    old = ops.set_kernel_family(family)
    try:
        got = ops.qk_forward(q, k, win, left, dil), ops.av_forward(attn, k, win, left, dil), ops.v_backward(attn, q, win, left, dil)
    finally:
        ops.set_kernel_family(old)
    eps = 2.0 ** -9 if dtype == torch.bfloat16 else 2.0 ** -12      # half a rounding step
    for i, (a, r) in enumerate(zip(got, _pair_reference(q, k, attn, win, left, dil))):
        rel = 2e-6 if i == 0 else eps * (1.1 if family in (0, 3, 4) else 1.6)
        assert float((a.double() - r).norm()) <= rel * float(r.norm()) + 1e-6, i


@pytest.mark.parametrize("C,routes", [(48, (3, 0)), (16, (4, 0))])
@pytest.mark.parametrize("value", [float("nan"), float("inf")])
def test_unfused_operators_keep_bad_values_in_their_window(value, C, routes):
    from pcf_nat_b200 import ops
    q, k, d_o, _, _, _ = _inputs((1, 1, 150, C, 9, 4, 1, True, False), torch.bfloat16)
    attn = torch.rand(1, 150, 9, device="cuda")
    for bad in (q, k, attn):
        x = [q.clone(), k.clone(), attn.clone()]
        x[[id(q), id(k), id(attn)].index(id(bad))][0, 70, 5] = value
        out = []
        for family in routes:
            old = ops.set_kernel_family(family)
            try:
                out.append([ops.qk_forward(x[0], x[1], 9, 4), ops.av_forward(x[2], x[1], 9, 4), ops.v_backward(x[2], x[0], 9, 4)])
            finally:
                ops.set_kernel_family(old)
        for a, b in zip(*out):
            assert torch.equal(torch.isfinite(a), torch.isfinite(b)) and torch.equal(torch.isnan(a), torch.isnan(b))
            ok = torch.isfinite(b)
            assert torch.allclose(a[ok].float(), b[ok].float(), rtol=1e-2, atol=1e-2)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("C", [24, 48, 128])
def test_bands_keep_all_their_bits(C, dtype):
    """Two band entries on equal rows that cancel but for the last bits of one of them: the remainder, 2^-23 of the entries, comes
    out whole, in every place of the 24 bits."""
    from pcf_nat_b200 import ops
    T, win = 40, 5
    x = torch.full((1, T, C), 1.5, device="cuda", dtype=dtype)
    bits = torch.arange(T, device="cuda") % 23 + 1                          # the bit that survives in row t
    band = torch.zeros(1, T, win, device="cuda")
    odd = 1 + 0.25 + 2.0 ** -9 + 2.0 ** -13                                 # pieces in between, none a power of two
    tail = torch.exp2(-bits.float())
    band[0, :, 2] = odd + tail
    band[0, :, 1] = -odd
    left = (band[0, :, 2].double() + band[0, :, 1].double()) * 1.5          # (key t - 1 + key t, both 1.5; row 0 has no key -1)
    old = ops.set_kernel_family(ops.FAMILY_WARP_MMA)
    try:
        av = ops.av_forward(band, x, win, 2)[0]
        vb = ops.v_backward(band, x, win, 2)[0]
    finally:
        ops.set_kernel_family(old)
    assert torch.equal(av[1:].double(), left[1:, None].to(dtype).double().expand(T - 1, C))
    want = (band[0, :, 2].double() + torch.cat([band[0, 1:, 1], band.new_zeros(1)]).double()) * 1.5     # key t: queries t and t + 1
    assert torch.equal(vb.double(), want[:, None].to(dtype).double().expand(T, C))


@pytest.mark.parametrize("scale", [1.0, 1e-6])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("N,T,C,win,dil", [(40, 20, 16, 17, 1), (40, 31, 64, 9, 1), (30, 21, 32, 27, 2), (20, 100, 64, 40, 1), (20, 150, 48, 50, 1), (20, 90, 128, 33, 3),
                                           (3000, 150, 16, 27, 1), (500, 150, 64, 33, 1)])
def test_unfused_routes_lose_no_bits_of_the_band(N, T, C, win, dil, dtype, scale):
    """Where the CUDA-core kernels stand in for shapes that tcgen05 does not take, the automatic route gives their fp32 products bit
    for bit, and results from a band (of gradients as small as an unscaled loss leaves them) that are no further from 64 bits."""
    from pcf_nat_b200 import ops
    g = torch.Generator(device="cuda").manual_seed(4)
    q, k = (torch.randn(N, T, C, device="cuda", generator=g).to(dtype) for _ in range(2))
    band = torch.randn(N, T, win, device="cuda", generator=g) * scale
    left = win // 2
    got = {}
    for family in (ops.FAMILY_AUTO, ops.FAMILY_CUDA_CORE):
        old = ops.set_kernel_family(family)
        try:
            got[family] = ops.qk_forward(q, k, win, left, dil), ops.av_forward(band, k, win, left, dil), ops.v_backward(band, q, win, left, dil)
        finally:
            ops.set_kernel_family(old)
    tcgen05 = C in (16, 32, 64) and T >= 32 and dil & (dil - 1) == 0 and (win - 1) * dil + 1 <= 33
    ref = _pair_reference(q, k, band, win, left, dil)
    if not tcgen05:
        assert torch.equal(got[ops.FAMILY_AUTO][0], got[ops.FAMILY_CUDA_CORE][0])
    for i in (1, 2):
        if tcgen05 and (i == 1 or dtype == torch.float16 and C == 64):
            continue                                  # (the tcgen05 kernels round the band to 16 bits)
        auto, core = (float((got[f][i].double() - ref[i]).norm()) for f in (ops.FAMILY_AUTO, ops.FAMILY_CUDA_CORE))
        # both round an fp32 result once; elements that round the other way scatter the norm
        assert auto <= core * (1 + 1e-4 + 0.02 / ref[i].numel() ** 0.5), (i, auto, core)
