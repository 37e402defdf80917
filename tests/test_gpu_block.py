"""The block's row and column kernels and the fused block node against plain PyTorch in 64 bits (or the same module run
part by part). Sizes sit at the edges: one row, row counts around a CTA's eight, rows of 8 channels, of one chunk of 256 and
one more, the largest of 1024; time axes shorter than the CTA's warps."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu

DT = [torch.bfloat16, torch.float16]
EPS = {torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11}    # rounding step of one 16-bit store


def _rand(*shape, dtype, seed, scale=1.0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return (torch.randn(*shape, device="cuda", generator=g) * scale).to(dtype)


def _close(got, ref, dtype, steps=1.0):
    """Within ``steps`` 16-bit rounding steps of the value, plus fp32 noise relative to the tensor's largest value."""
    err = (got.double() - ref).abs()
    bound = steps * EPS[dtype] * ref.abs() + 4e-6 * ref.abs().max() + 1e-7
    assert bool((err <= bound).all()), float((err - bound).max())


@pytest.mark.parametrize("dtype", DT)
@pytest.mark.parametrize("rows,D", [(1, 8), (7, 64), (8, 256), (9, 264), (300, 256), (5000, 192), (33, 512), (17, 776), (20, 1024)])
def test_layer_norm_with_residual(rows, D, dtype):
    import block_passes as block
    x, dx, dy, res = (_rand(rows, D, dtype=dtype, seed=s) for s in range(4))
    w, b = 1 + _rand(D, dtype=torch.float32, seed=5, scale=0.2), _rand(D, dtype=torch.float32, seed=6, scale=0.2)
    y, s, mean, rstd = block.layer_norm(x, dx, w, b, 1e-5, True)
    assert torch.equal(s, x + dx)
    s64, w64, b64 = s.double().requires_grad_(), w.double().requires_grad_(), b.double().requires_grad_()
    ref = F.layer_norm(s64, (D,), w64, b64, 1e-5)
    _close(y, ref.detach(), dtype)
    y0, s0, none, _ = block.layer_norm(s, None, w, b, 1e-5, False)
    assert torch.equal(y0, y) and s0 is s and none is None
    for r in (res, None):
        ds, sums = block.layer_norm_backward(dy, s, mean, rstd, w, r, block.scratch_for(rows, D, 8, x.device))
        gs, gw, gb = torch.autograd.grad(ref, (s64, w64, b64), dy.double(), retain_graph=True)
        gs = gs if r is None else gs + r.double()
        # the row sums cancel: fp32 noise of the terms, not of the result
        err = (ds.double() - gs).abs()
        assert bool((err <= EPS[dtype] * gs.abs() + 2e-5 * float(dy.double().abs().max() * rstd.max())).all())
        for got, want, terms in ((sums[0], gw, rows ** 0.5), (sums[1], gb, rows ** 0.5), (sums[2], ds.double().sum(0), rows ** 0.5)):
            assert float((got.double() - want).abs().max()) <= 1e-5 * (terms + 3) * 4


@pytest.mark.parametrize("dtype", DT)
@pytest.mark.parametrize("rows,F_", [(1, 8), (9, 256), (700, 264), (4099, 1024), (65, 2048)])
def test_gelu_and_column_sums(rows, F_, dtype):
    import block_passes as block
    x, dy = _rand(rows, F_, dtype=dtype, seed=1, scale=2.0), _rand(rows, F_, dtype=dtype, seed=2)
    x64 = x.double().requires_grad_()
    ref = F.gelu(x64)
    got = block.gelu(x)
    # half a rounding step, and the approximation's 0.75e-7 |x| (fp16 subnormals: their own spacing)
    bound = EPS[dtype] * ref.detach().abs() + 2e-7 * x64.detach().abs() + (6e-8 if dtype == torch.float16 else 0)
    assert bool(((got.double() - ref.detach()).abs() <= bound).all())
    torch_err = (F.gelu(x).double() - ref.detach()).norm()
    assert float((got.double() - ref.detach()).norm()) <= 1.001 * float(torch_err)      # no less exact than the framework's
    scratch = block.scratch_for(rows, 8, F_, x.device)
    dx, sums = block.gelu_backward(dy, x, scratch)
    want = torch.autograd.grad(ref, x64, dy.double())[0]
    _close(dx, want, dtype)
    assert float((sums.double() - dx.double().sum(0)).abs().max()) <= 1e-5 * (rows ** 0.5 + 3)
    assert float((block.column_sums(dy, scratch).double() - dy.double().sum(0)).abs().max()) <= 1e-5 * (rows ** 0.5 + 3)


def test_gelu_of_special_values():
    import block_passes as block
    for dtype in DT:
        x = torch.tensor([0.0, -0.0, float("inf"), float("-inf"), float("nan"), 3e4, -3e4, -8.0], device="cuda", dtype=dtype)
        got, ref = block.gelu(x).float(), F.gelu(x).float()
        assert torch.equal(torch.isnan(got), torch.isnan(ref))
        ok = ~torch.isnan(ref)
        assert torch.allclose(got[ok], ref[ok], rtol=1e-2, atol=1e-6)


def test_cast_parameters_is_the_rounding_of_each_tensor():
    import block_passes as block
    for dtype in DT:
        ps = [_rand(n, dtype=torch.float32, seed=n) for n in (1, 7, 8, 63, 64, 2048, 2049, 70001)]
        ps.append(_rand(33, dtype=torch.float32, seed=3)[1:])          # not 16-byte aligned
        buf, offs = block.cast_parameters(ps, dtype)
        for p, o in zip(ps, offs):
            assert torch.equal(buf[o:o + p.numel()], p.to(dtype))


@pytest.mark.parametrize("dtype", DT)
@pytest.mark.parametrize("N,T,C", [(1, 1, 8), (2, 7, 256), (3, 9, 264), (5, 300, 1536), (2, 1000, 40)])
def test_statistics_pooling(N, T, C, dtype):
    from pcf_nat_b200 import block
    logits, x = _rand(N, T, C, dtype=dtype, seed=1, scale=3.0).requires_grad_(), _rand(N, T, C, dtype=dtype, seed=2).requires_grad_()
    d_out = _rand(N, 2 * C, dtype=torch.float32, seed=3)
    out = block.stats_pool(logits, x, 1e-5)
    l64, x64 = logits.detach().double().requires_grad_(), x.detach().double().requires_grad_()
    w = torch.softmax(l64, 1)
    mu = (w * x64).sum(1)
    var = (w * x64 * x64).sum(1) - mu * mu
    ref = torch.cat([mu, var.clamp_min(1e-5).sqrt()], 1)
    mean_ref, std_ref, var = ref[:, :C].detach(), ref[:, C:].detach(), var.detach()
    assert float((out[:, :C].detach().double() - mean_ref).abs().max()) <= 2e-5
    # the variance is a difference of two fp32 sums: 4e-6 of it, through the square root
    assert bool(((out[:, C:].detach().double() - std_ref).abs() <= 4e-6 * (1 + mean_ref ** 2) / std_ref + 1e-6).all())
    clear = (var > 1e-3)                      # away from the floor, where the gradient of the square root is steep
    d_out[:, C:] *= clear
    g = torch.autograd.grad(out, (logits, x), d_out)
    r = torch.autograd.grad(ref, (l64, x64), d_out.double())
    for got, want in zip(g, r):
        err = float((got.double() - want).norm()), float(want.norm())
        assert err[0] <= (EPS[dtype] + 2e-4) * err[1] + 1e-6, err


def test_pooling_with_infinite_logits_and_a_constant_channel():
    from pcf_nat_b200 import block
    logits = torch.zeros(1, 20, 8, device="cuda", dtype=torch.bfloat16)
    x = _rand(1, 20, 8, dtype=torch.bfloat16, seed=1)
    logits[0, :10, 0] = float("-inf")          # half of the frames have no weight
    logits[0, :, 1] = float("-inf")            # none has: 0 / 0
    logits[0, 3, 2] = float("inf")
    logits[0, 3, 3] = float("nan")
    logits[0, :, 4] = -3e38
    x[0, :, 5] = 1.0                           # variance 0: the floor
    w = torch.softmax(logits.float(), 1)
    mu = (w * x.float()).sum(1)
    ref = torch.cat([mu, ((w * x.float() ** 2).sum(1) - mu * mu).clamp_min(1e-5).sqrt()], 1)
    assert torch.allclose(block.stats_pool(logits, x, 1e-5), ref, rtol=1e-5, atol=1e-5, equal_nan=True)


def _stage(dim, heads, frames, hidden=4, n=2):
    from pcf_nat_b200.model import NABlock
    torch.manual_seed(3)
    return torch.nn.ModuleList(NABlock(frames, dim, heads, 7, hidden, "fused") for _ in range(n)).cuda()


@pytest.mark.parametrize("dtype", DT)
@pytest.mark.parametrize("dim,heads,T", [(64, 2, 50), (256, 4, 131), (512, 8, 40)])
def test_block_node_against_its_modules(dim, heads, T, dtype):
    """Outputs and all gradients of the fused node, of the module-by-module network and of the same network in fp32: the node
    is no further from fp32 than the modules are."""
    from pcf_nat_b200 import block
    st = _stage(dim, heads, T)
    x0 = _rand(3, T, dim, dtype=dtype, seed=1)
    dy = _rand(3, T, dim, dtype=dtype, seed=2)
    got = {}
    for kind in ("node", "modules"):
        x = x0.clone().requires_grad_()
        with torch.autocast("cuda", dtype=dtype):
            if kind == "node":
                y = block.run_blocks(st, x, None)
                assert y is not None
            else:
                y = x
                for b in st:
                    y = b(y)
        got[kind] = [y.detach()] + list(torch.autograd.grad(y, [x] + list(st.parameters()), dy))
    ref = _reference(st, x0, dy, heads)
    for a, b, r in zip(got["node"], got["modules"], ref):
        assert a.dtype == b.dtype and a.shape == b.shape
        ea, eb = float((a.double() - r).norm()), float((b.double() - r).norm())
        # the norm of n independent rounding errors scatters by 1 / sqrt(2 n) of itself: four times that for the two of them
        n = r.numel()
        assert ea <= (1.1 + 4 / n ** 0.5) * eb + 1e-6 * float(r.norm()), (ea, eb, float(r.norm()), tuple(r.shape))


def _reference(st, x0, dy, heads):
    from oracle import na1d_oracle as orc
    w = [p.detach().double().cpu().requires_grad_() for p in st.parameters()]
    named = dict(zip([n for n, _ in st.named_parameters()], w))
    x = x0.double().cpu().requires_grad_()
    y = x
    B, T, D = x.shape
    C = D // heads
    for i in range(len(st)):
        p = {n[2:]: v for n, v in named.items() if n.startswith("%d." % i)}
        h = F.layer_norm(y, (D,), p["norm1.weight"], p["norm1.bias"])
        q, k, v = F.linear(h, p["attn.qkv.weight"], p["attn.qkv.bias"]).view(B, T, 3, heads, C).permute(2, 0, 3, 1, 4).reshape(3, B * heads, T, C)
        o = orc.na1d_fused(q, k, v, 7, 3, 1, C ** -0.5, p["attn.relative_position_bias"].view(heads, 7), None, heads)
        o = o.view(B, heads, T, C).transpose(1, 2).reshape(B, T, D)
        y = y + F.linear(o, p["attn.proj.weight"], p["attn.proj.bias"])
        h = F.layer_norm(y, (D,), p["norm2.weight"], p["norm2.bias"])
        y = y + F.linear(F.gelu(F.linear(h, p["fc1.weight"], p["fc1.bias"])), p["fc2.weight"], p["fc2.bias"])
    g = torch.autograd.grad(y, [x] + w, dy.double().cpu())
    return [t.detach().cuda() for t in (y,) + g]


def test_block_node_evaluation_with_padding_and_frozen_parameters():
    from pcf_nat_b200 import block
    from pcf_nat_b200.nattention import _valid_tokens
    st = _stage(128, 4, 60).eval()
    x = _rand(3, 60, 128, dtype=torch.bfloat16, seed=1)
    pad = torch.tensor([0, 13, 60], device="cuda")
    with torch.no_grad(), torch.autocast("cuda", dtype=torch.bfloat16):
        y = block.run_blocks(st, x, _valid_tokens(60, pad, 3))
        z = x
        for b in st:
            z = b(z, pad)
    assert float((y.double() - z.double()).norm() / z.double().norm()) < 1e-2
    st.train()
    for n, p in st.named_parameters():
        p.requires_grad_("fc1" in n)
    with torch.autocast("cuda", dtype=torch.bfloat16):
        y = block.run_blocks(st, x, None)
    y.float().sum().backward()
    assert all((p.grad is not None) == ("fc1" in n) for n, p in st.named_parameters())


def test_block_node_leaves_other_blocks_to_their_modules():
    from pcf_nat_b200 import block
    x = _rand(2, 40, 64, dtype=torch.bfloat16, seed=1)

    def refused(change, x=x, enabled=True):
        st = _stage(64, 2, 40)
        change(st)
        with torch.autocast("cuda", dtype=torch.bfloat16, enabled=enabled):
            return block.run_blocks(st, x, None) is None

    assert not refused(lambda st: None)
    assert refused(lambda st: None, enabled=False)
    assert refused(lambda st: None, x=x.float())
    assert refused(lambda st: st[1].fc1.register_forward_hook(lambda *a: None))
    assert refused(lambda st: st.bfloat16())
    assert refused(lambda st: setattr(st[0].attn.proj_drop, "p", 0.1))
    assert refused(lambda st: setattr(st[0], "norm1", torch.nn.LayerNorm(64, bias=False).cuda()))
    assert refused(lambda st: setattr(st[0], "fc2", torch.nn.Sequential(st[0].fc2)))


@pytest.mark.parametrize("dtype", DT)
@pytest.mark.parametrize("N,C,T", [(1, 8, 1), (2, 64, 64), (3, 72, 65), (2, 256, 150), (2, 136, 97), (1, 64, 2)])
def test_transpose(N, C, T, dtype):
    from pcf_nat_b200 import _lib, ops
    code = _lib.NA1D_BF16 if dtype == torch.bfloat16 else _lib.NA1D_FP16
    for off in (0, 1):                       # an odd base cannot be read in pairs
        x = _rand(N * C * T + 1, dtype=dtype, seed=1)[off:off + N * C * T].view(N, C, T)
        y, z = torch.empty(N, T, C, device="cuda", dtype=dtype), torch.full((N * C * T + 1,), 7.0, device="cuda", dtype=dtype)
        s = torch.cuda.current_stream().cuda_stream
        assert ops._L.na1d_transpose(y.data_ptr(), x.data_ptr(), N, C, T, 1, code, s) == 0
        assert torch.equal(y, x.transpose(1, 2))
        assert ops._L.na1d_transpose(z[off:].data_ptr(), y.data_ptr(), N, C, T, 0, code, s) == 0
        assert torch.equal(z[off:off + N * C * T].view(N, C, T), x) and float(z[-1 if off == 0 else 0]) == 7.0


@pytest.mark.parametrize("autocast", [True, False])
@pytest.mark.parametrize("layout,groups,dim,heads,T,bias", [("channels_first", 8, 128, 8, 150, True), ("channels_first", 1, 64, 1, 77, False),
                                                            ("channels_first", 2, 192, 4, 65, True), ("channels_last", 1, 256, 8, 51, True),
                                                            ("channels_last", 1, 64, 2, 64, False), ("channels_last", 1, 96, 2, 53, True)])
def test_layer_node_against_the_layer_in_fp32(layout, groups, dim, heads, T, bias, autocast):
    """Output and every gradient of the layer in 16 bits against its own parameters and input in 64 bits: four rounding steps of
    the intermediate tensors, relative to each result."""
    from oracle import na1d_oracle as orc
    from pcf_nat_b200 import NAttention, ops
    torch.manual_seed(5)
    m = NAttention(T, dim, heads, 9, 1, groups, layout=layout, qkv_bias=bias, proj_bias=bias).cuda()
    if not autocast:
        m = m.to(torch.float16)
    dt = torch.bfloat16 if autocast else torch.float16
    first = layout == "channels_first"
    x = _rand(*((2, dim, T) if first else (2, T, dim)), dtype=dt, seed=1).requires_grad_()
    dy = _rand(*x.shape, dtype=dt, seed=2)
    with torch.autocast("cuda", dtype=torch.bfloat16, enabled=autocast):
        y = m(x)
    # (48 and 64 channels, 65 and 77 tokens, below: one size the packed route takes in each layout, one it does not)
    assert "NA1dLayer" in y.grad_fn.name()
    if dim // heads == 48:
        assert not ops.packed_supported(heads, T, 48, 9, 4, 1, dt)
    ps = dict(m.named_parameters())
    got = [y.detach()] + list(torch.autograd.grad(y, [x] + list(ps.values()), dy))
    w = {n: p.detach().double().cpu().requires_grad_() for n, p in ps.items()}
    x64 = x.detach().double().cpu().requires_grad_()
    C = dim // heads
    if first:
        h = F.conv1d(x64, w["qkv.weight"], w.get("qkv.bias"), groups=groups)
        h = h.view(2, dim // groups, groups, 3, T).transpose(1, 2).reshape(2, heads, C, 3, T).permute(3, 0, 1, 4, 2)
    else:
        h = F.linear(x64, w["qkv.weight"], w.get("qkv.bias")).view(2, T, 3, heads, C).permute(2, 0, 3, 1, 4)
    q, k, v = h.reshape(3, 2 * heads, T, C)
    o = orc.na1d_fused(q, k, v, 9, 4, 1, C ** -0.5, w["relative_position_bias"].view(heads, 9), None, heads).view(2, heads, T, C)
    if first:
        ref = F.conv1d(o.transpose(2, 3).reshape(2, dim, T), w["proj.weight"], w.get("proj.bias"), groups=groups)
    else:
        ref = F.linear(o.transpose(1, 2).reshape(2, T, dim), w["proj.weight"], w.get("proj.bias"))
    want = [ref.detach()] + list(torch.autograd.grad(ref, [x64] + list(w.values()), dy.double().cpu()))
    for name, a, r in zip(["y", "x"] + list(w), got, want):
        assert a.shape == r.shape and a.dtype == (dt if name in ("y", "x") or not autocast else torch.float32)
        assert float((a.double().cpu() - r).norm()) <= 4 * EPS[dt] * float(r.norm()) + 1e-6, name


@pytest.mark.parametrize("B,T,parts,H,C", [(1, 1, 1, 1, 8), (2, 65, 3, 4, 48), (3, 7, 1, 5, 128), (2, 300, 3, 2, 64)])
def test_permute_heads(B, T, parts, H, C):
    from pcf_nat_b200 import ops
    x = _rand(B, T, parts, H, C, dtype=torch.bfloat16, seed=1)
    y, z = torch.empty(parts, B, H, T, C, device="cuda", dtype=x.dtype), torch.empty_like(x)
    s = torch.cuda.current_stream().cuda_stream
    assert ops._L.na1d_permute_heads(y.data_ptr(), x.data_ptr(), B, T, parts, H, C, 1, s) == 0
    assert torch.equal(y, x.permute(2, 0, 3, 1, 4))
    assert ops._L.na1d_permute_heads(z.data_ptr(), y.data_ptr(), B, T, parts, H, C, 0, s) == 0
    assert torch.equal(z, x)


def test_layer_node_leaves_mixed_types_and_hooks_alone():
    from pcf_nat_b200 import NAttention
    for layout in ("channels_first", "channels_last"):
        m = NAttention(64, 64, 2, 7, layout=layout).cuda()
        x = _rand(2, 64, 64, dtype=torch.bfloat16, seed=1)
        with pytest.raises(RuntimeError):
            m(x)                                                        # fp32 weights without autocast
        with torch.autocast("cuda", dtype=torch.float16):
            assert m(x).dtype == torch.float16                          # autocast's type wins over the input's
    seen = []
    m.qkv.register_forward_hook(lambda *a: seen.append(1))
    with torch.autocast("cuda", dtype=torch.bfloat16):
        m(x)
    assert seen == [1]


@pytest.mark.parametrize("dtype", DT)
def test_rows_written_into_their_slice(dtype):
    from pcf_nat_b200 import block
    x, dx = _rand(3, 17, 72, dtype=dtype, seed=1), _rand(3, 17, 72, dtype=dtype, seed=2)
    with torch.no_grad():
        rows = block.feature_rows(x, 3)
    rows.fill_(7.0)
    block.add_to_rows(rows[..., 72:144], x, dx)
    assert torch.equal(rows[..., 72:144], x + dx) and bool((rows[..., :72] == 7).all()) and bool((rows[..., 144:] == 7).all())
    block.add_to_rows(rows[..., :72], x)
    assert torch.equal(rows[..., :72], x)
    logits = _rand(3, 17, 144, dtype=dtype, seed=3)
    with torch.no_grad():
        assert torch.equal(block.stats_pool(logits, rows[..., :144], 1e-5), block.stats_pool(logits, rows[..., :144].contiguous(), 1e-5))
    assert block.feature_rows(x, 3) is None                     # gradients on: the stages' outputs stay tensors of their own


def test_evaluation_with_shared_rows_gives_the_bits_of_separate_tensors(monkeypatch):
    from pcf_nat_b200 import block
    from pcf_nat_b200.model import PCFNATExtractor
    torch.manual_seed(2)
    m = PCFNATExtractor(frames=70, feat=24, dim=64, heads=2, win=7, stages=3, blocks=2, emb=32, classes=40).cuda().eval()
    x = _rand(4, 24, 70, dtype=torch.float32, seed=1)
    pad = torch.tensor([0, 3, 30, 7], device="cuda")
    with torch.no_grad(), torch.autocast("cuda", dtype=torch.bfloat16):
        a = m.embedding(x, pad)
        monkeypatch.setattr(block, "feature_rows", lambda *_: None)
        b = m.embedding(x, pad)
        m.stages[1][0].fc1.register_forward_hook(lambda *_: None)      # a stage that runs module by module in between
        monkeypatch.undo()
        c = m.embedding(x, pad)
    # (a GEMM on strided rows may pick another kernel: the last 16-bit rounding can differ)
    for other in (a, c):
        assert float((other.double() - b.double()).norm()) <= 2e-2 * float(b.double().norm())


def test_padding_lengths_may_live_on_the_host():
    """Lengths on the host or of another integer type give the bits of int32 lengths on the device, in the blocks and in the
    whole network; lengths for another number of utterances are left to the modules, which refuse them."""
    from pcf_nat_b200 import block
    from pcf_nat_b200.model import PCFNATExtractor
    st = _stage(64, 2, 50).eval()
    x = _rand(3, 50, 64, dtype=torch.bfloat16, seed=1)
    valid = torch.tensor([50, 17, 0], dtype=torch.int32)
    with torch.no_grad(), torch.autocast("cuda", dtype=torch.bfloat16):
        want = block.run_blocks(st, x, valid.cuda())
        assert not torch.equal(want, block.run_blocks(st, x, None))
        for v in (valid, valid.long(), valid.long().cuda(), valid.repeat_interleave(2)[::2]):
            assert torch.equal(block.run_blocks(st, x, v), want)
        assert block.run_blocks(st, x, valid[:2]) is None
    torch.manual_seed(2)
    m = PCFNATExtractor(frames=70, feat=24, dim=64, heads=2, win=7, stages=2, blocks=1, emb=32, classes=40).cuda().eval()
    fbank, pad = _rand(4, 24, 70, dtype=torch.float32, seed=1), torch.tensor([0, 3, 30, 7])
    with torch.no_grad(), torch.autocast("cuda", dtype=torch.bfloat16):
        assert torch.equal(m.embedding(fbank, pad), m.embedding(fbank, pad.cuda()))
        assert not torch.equal(m.embedding(fbank, pad), m.embedding(fbank))


def _second(y, x, params):
    """Gradients of a penalty on the input gradient, and that gradient."""
    g, = torch.autograd.grad(y.float().pow(2).sum(), x, create_graph=True)
    out = torch.autograd.grad(g.float().pow(2).sum(), [x] + params, allow_unused=True)
    return [g.detach()] + [torch.zeros_like(p) if o is None else o for o, p in zip(out, [x] + params)]


def _same(got, want, bound):
    for i, (a, b) in enumerate(zip(got, want)):
        assert a.dtype == b.dtype and a.shape == b.shape
        assert float((a.double() - b.double()).norm()) <= bound * float(b.double().norm()) + 1e-6, i


@pytest.mark.parametrize("chained", [False, True])
def test_second_derivative_of_blocks(chained):
    """A gradient penalty through one block, or through two with the sum between them inside the second, with some parameters
    frozen: the one-node route gives what the modules give (eight rounding steps of bf16 for the chain of about that many
    16-bit tensors; a lost term would be of the order of the result)."""
    from pcf_nat_b200 import block
    st = _stage(64, 2, 40, n=2 if chained else 1)
    for n, p in st.named_parameters():
        p.requires_grad_("norm1.bias" not in n)
    params = [p for p in st.parameters() if p.requires_grad]
    got = {}
    for kind in ("node", "modules"):
        x = _rand(2, 40, 64, dtype=torch.bfloat16, seed=1, scale=0.5).requires_grad_()
        with torch.autocast("cuda", dtype=torch.bfloat16):
            y = block.run_blocks(st, 2 * x, None) if kind == "node" else 2 * x
            for b in st if kind == "modules" else ():
                y = b(y)
        got[kind] = _second(y, x, params)
    _same(got["node"], got["modules"], 8 * EPS[torch.bfloat16])


@pytest.mark.parametrize("autocast", [True, False])
@pytest.mark.parametrize("layout,groups,dim,heads,bias", [("channels_first", 4, 128, 4, True), ("channels_last", 1, 64, 2, False), ("channels_last", 1, 96, 2, True)])
def test_second_derivative_of_a_layer(layout, groups, dim, heads, bias, autocast):
    from pcf_nat_b200 import NAttention, nattention
    torch.manual_seed(5)
    m = NAttention(50, dim, heads, 9, 1, groups, layout=layout, qkv_bias=bias, proj_bias=bias).cuda()
    m = m if autocast else m.half()
    got = {}
    for kind in ("node", "modules"):
        x = _rand(*((2, dim, 50) if layout == "channels_first" else (2, 50, dim)), dtype=torch.float16, seed=1).requires_grad_()
        with torch.autocast("cuda", dtype=torch.float16, enabled=autocast), pytest.MonkeyPatch.context() as mp:
            if kind == "modules":
                mp.setattr(nattention, "_native_layer", lambda *a: None)
            y = m(1 * x)
        assert ("NA1dLayer" in y.grad_fn.name()) == (kind == "node")
        got[kind] = _second(y, x, list(m.parameters()))
    _same(got["node"], got["modules"], 8 * EPS[torch.float16])


def test_second_derivative_of_the_pooling():
    from pcf_nat_b200 import block
    logits, x = _rand(2, 30, 16, dtype=torch.float16, seed=1).requires_grad_(), _rand(2, 30, 16, dtype=torch.float16, seed=2)
    x[:, :, 3] = 1.0                              # variance 0: the floor
    x.requires_grad_()
    got = []
    for pool in (block.stats_pool, block.weighted_stats):
        out = pool(logits * 1, x * 1, 1e-5)
        g = torch.autograd.grad(out.pow(2).sum(), (logits, x), create_graph=True)
        got.append([t.detach() for t in g] + list(torch.autograd.grad(sum(t.float().pow(2).sum() for t in g), (logits, x))))
    _same(got[0], got[1], 4 * EPS[torch.float16])


@pytest.mark.parametrize("kind", ["block", "channels_first", "channels_last"])
def test_backward_under_autocast_keeps_the_types_of_the_forward(kind):
    from pcf_nat_b200 import NAttention, block
    torch.manual_seed(5)
    m = _stage(64, 2, 40, n=1) if kind == "block" else NAttention(40, 64, 2, 7, layout=kind).cuda()
    x = _rand(*((2, 64, 40) if kind == "channels_first" else (2, 40, 64)), dtype=torch.bfloat16, seed=1).requires_grad_()
    with torch.autocast("cuda", dtype=torch.bfloat16):
        y = block.run_blocks(m, x, None) if kind == "block" else m(x)
    ins, dy = [x] + list(m.parameters()), _rand(*y.shape, dtype=torch.bfloat16, seed=2)
    want = torch.autograd.grad(y, ins, dy, retain_graph=True)
    for dtype in DT:
        with torch.autocast("cuda", dtype=dtype):
            got = torch.autograd.grad(y, ins, dy, retain_graph=True)
        for a, b in zip(got, want):
            assert a.dtype == b.dtype and torch.allclose(a, b, rtol=1e-4, atol=1e-4)      # (atomics in the bias table's gradient)


@pytest.mark.parametrize("kind", ["block", "channels_first", "channels_last"])
def test_output_gradients_may_start_anywhere(kind):
    """A contiguous view that is not on a 16-byte boundary gives the gradients of its aligned copy."""
    from pcf_nat_b200 import NAttention, block
    torch.manual_seed(5)
    m = _stage(64, 2, 40, n=1) if kind == "block" else NAttention(40, 64, 2, 7, layout=kind).cuda()
    x = _rand(*((2, 64, 40) if kind == "channels_first" else (2, 40, 64)), dtype=torch.bfloat16, seed=1).requires_grad_()
    with torch.autocast("cuda", dtype=torch.bfloat16):
        y = block.run_blocks(m, 1 * x, None) if kind == "block" else m(1 * x)
    ins, dy = [x] + list(m.parameters()), _rand(y.numel() + 1, dtype=torch.bfloat16, seed=2)[1:].view(y.shape)
    assert dy.is_contiguous() and dy.data_ptr() % 16
    for a, b in zip(torch.autograd.grad(y, ins, dy, retain_graph=True), torch.autograd.grad(y, ins, dy.clone(), retain_graph=True)):
        assert torch.allclose(a, b, rtol=1e-4, atol=1e-4)      # (atomics in the bias table's gradient)


def test_layers_longer_than_the_transposes_take_run():
    from pcf_nat_b200 import NAttention
    T = 2 ** 20 + 8
    m = NAttention(8, 16, 1, 3, layout="channels_first").cuda().half()
    x = _rand(1, 16, T, dtype=torch.float16, seed=1).requires_grad_()
    y = m(x)
    assert "NA1dLayer" not in y.grad_fn.name()
    dx, = torch.autograd.grad(y, x, torch.ones_like(y))
    with torch.no_grad():
        part = m(x[..., -500:].contiguous())
    assert torch.allclose(y[..., -499:], part[..., 1:], rtol=4 * EPS[x.dtype], atol=1e-3) and bool(torch.isfinite(dx).all())


@pytest.mark.parametrize("layout", ["channels_first", "channels_last"])
def test_layer_without_a_bias_table(layout):
    from pcf_nat_b200 import NAttention
    m = NAttention(64, 64, 2, 7, layout=layout).cuda().half()
    x = _rand(2, 64, 64, dtype=torch.float16, seed=1)
    with torch.no_grad():
        m.relative_position_bias.zero_()
        want = m(x)
        m.relative_position_bias = None
        assert torch.allclose(m(x), want, rtol=4 * EPS[torch.float16], atol=1e-3)


@pytest.mark.parametrize("dtype", DT)
def test_gelu_of_every_16_bit_value(dtype):
    """Against 64 bits: no more results, and no more between -4 and 4, round the wrong way than the framework's, in the function
    and in its derivative (five values to spare: both are off by rounding errors of fp32 alone there)."""
    import block_passes as block
    x = torch.arange(-32768, 32768, device="cuda", dtype=torch.int32).to(torch.int16).view(dtype)
    x = x[torch.isfinite(x)]
    x = x[:x.numel() // 8 * 8].clone()
    x64, xf, one = x.double().requires_grad_(), x.clone().requires_grad_(), torch.ones_like(x)
    ref, theirs = F.gelu(x64), F.gelu(xf)
    d_ref, d_theirs = torch.autograd.grad(ref, x64, one.double())[0], torch.autograd.grad(theirs, xf, one)[0]
    ours, (d_ours, _) = block.gelu(x), block.gelu_backward(one.view(-1, 8), x.view(-1, 8), block.scratch_for(x.numel() // 8, 8, 8, x.device))
    near = x.float().abs() < 4
    for a, b, r in ((ours, theirs, ref), (d_ours.view(-1), d_theirs, d_ref)):
        wrong = [t.detach() != r.detach().to(dtype) for t in (a, b)]
        assert int(wrong[0].sum()) <= int(wrong[1].sum())
        assert int((wrong[0] & near).sum()) <= int((wrong[1] & near).sum()) + 5
