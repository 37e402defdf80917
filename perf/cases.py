"""The work that programs built on this package have it do, as timed cases.

Four kinds, all through the package's public entry points:

* ``op``    the fused operator ``na1d_fused`` -- forward alone under ``no_grad`` (inference) or forward and backward;
* ``pair``  the drop-in ``getNA1dFunction`` pair inside the eager chain of an unmodified model file: q*scale -> QK -> +bias ->
            +mask -> softmax -> AV, forward and backward;
* ``layer`` the packaged ``NAttention`` layer, channels-first (PCF) or channels-last (MFA), training or evaluation with padding;
* ``model`` the ``PCFNATExtractor`` network, a training step's forward and backward or the extraction of embeddings.

``listed()`` is the set that is followed over time; ``draw()`` samples the ranges those cases stand for.
"""
import math

import torch
import torch.nn.functional as F

from pcf_nat_b200 import NAttention, getNA1dFunction, na1d_fused
from pcf_nat_b200 import ops
from pcf_nat_b200.model import PCFNATExtractor, model_flops_per_utterance
from pcf_nat_b200.nattention import padding_mask
from pcf_nat_b200.parallel import flat_gradient_buffer

DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16}
FEAT, CLASSES = 80, 5994          # log-mel bins, speakers (the benchmark's extractor)
OP_ELEMENTS = 128 * 3000 * 64     # largest tensor of the operator cases, in elements
OP_PRODUCTS = 8192 * 150 * 27 * 16 * 1.5   # and largest number of (query, neighbour, channel) products
LAYER_ELEMENTS = 512 * 150 * 256  # largest layer input


def _op(name, batch, heads, T, C, win, train, left=None, dil=1, dtype="bf16", bias=False, padded=False, drop=0.0):
    left = win - 1 - win // 2 if left is None else left
    return {"name": name, "kind": "op", "batch": batch, "heads": heads, "T": T, "C": C, "win": win, "left": left, "dil": dil,
            "dtype": dtype, "bias": bias, "padded": padded, "drop": drop, "train": train}


def _layer(name, layout, batch, T, dim, heads, win, groups, train, dtype, dil=1):
    return {"name": name, "kind": "layer", "layout": layout, "batch": batch, "T": T, "dim": dim, "heads": heads, "win": win,
            "groups": groups, "dil": dil, "dtype": dtype, "train": train}


def _model(name, batch, frames, heads, win, train):
    return {"name": name, "kind": "model", "batch": batch, "frames": frames, "heads": heads, "win": win, "train": train}


def listed():
    return [
        # Scoring one pair of short utterances: the smallest call, bound by the latency of one launch.
        _op("op_infer_small", 2, 4, 200, 32, 7, False),
        # The training shape the operator is quoted on: 128 utterances of 2 s, 4 heads of 64 channels, window 7.
        _op("op_train", 128, 4, 200, 64, 7, True),
        # The reference's own configuration: 512 crops of 150 tokens, 16 heads of 16 channels, window 27, with the layer's
        # relative position bias and its gradient.
        _op("op_train_narrow", 512, 16, 150, 16, 27, True, bias=True),
        # Embedding extraction from 30 s utterances of different lengths, in fp16: forward only, padded batch.
        _op("op_infer_long", 16, 8, 3000, 64, 15, False, dtype="fp16", padded=True),
        # Wide dilated windows on ragged 10 s crops (the sweep's far corner; an odd number of tokens), fp16.
        _op("op_train_dilated", 64, 4, 997, 32, 31, True, dil=2, dtype="fp16"),
        # A layer whose head size and window are outside the tuned ones (the layer takes any multiple of 8 channels and
        # windows up to 80), with bias and padded utterances.
        _op("op_train_general", 64, 4, 203, 48, 41, True, bias=True, padded=True),
        # Training with attention dropout.
        _op("op_train_dropout", 64, 4, 299, 32, 15, True, bias=True, drop=0.1),
        # An unmodified model file that only swaps its import, at the reference's own configuration.
        {"name": "pair_train", "kind": "pair", "batch": 512, "heads": 16, "T": 150, "C": 16, "win": 27, "dil": 1, "dtype": "bf16"},
        # One layer of the reference's PCF model in a training step: 512 crops, grouped projections, bf16 autocast.
        _layer("layer_pcf_train", "channels_first", 512, 150, 256, 16, 27, 8, True, "autocast"),
        # One layer of the MFA model while it scores the 400-frame slices of an utterance, fp16 weights.
        _layer("layer_mfa_infer", "channels_last", 12, 200, 256, 16, 27, 1, False, "fp16"),
        # The extractor's training step on half a GPU's batch: forward and backward, gradients in one flat buffer.
        _model("model_train", 128, 300, 4, 7, True),
        # Embedding extraction, one batch of the extraction loop: 2-3 s utterances, padding masks.
        _model("model_infer", 512, 300, 4, 7, False),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choices(["op", "pair", "layer", "model"], [10, 2, 4, 2])[0]
    if kind == "op":
        C = rng.choice([16, 32, 64, 16, 32, 64, 16, 32, 64, 8, 24, 48, 96, 128])
        heads = rng.choice([1, 2, 4, 8, 16])
        win = _log_int(rng, 3, 80) if rng.random() < 0.4 else _log_int(rng, 3, 33)
        left = win - 1 - win // 2 if rng.random() < 0.8 else rng.randrange(win)
        dil = rng.choice([1, 1, 1, 1, 1, 2, 3, 4])
        T = _log_int(rng, 20, 3000)
        per_utterance = heads * T * C
        batch = _log_int(rng, 1, max(1, min(512, OP_ELEMENTS // per_utterance, int(OP_PRODUCTS // (per_utterance * win)))))
        train = rng.random() < 0.65
        drop = 0.1 if train and rng.random() < 0.25 and ops.dropout_supported(heads, T, C, win, dil) else 0.0
        case = _op("", batch, heads, T, C, win, train, left, dil, rng.choice(["bf16", "bf16", "fp16"]), rng.random() < 0.6,
                   rng.random() < 0.4, drop)
    elif kind == "pair":
        C, heads, win, T = rng.choice([16, 32, 64]), rng.choice([4, 8, 16]), _log_int(rng, 3, 33), _log_int(rng, 40, 1000)
        per_utterance = heads * T * max(C, win)
        batch = _log_int(rng, 1, max(1, min(512, 8192 * 150 * 27 // per_utterance)))
        case = {"kind": "pair", "batch": batch, "heads": heads, "T": T, "C": C, "win": win, "dil": 1,
                "dtype": rng.choice(["bf16", "bf16", "fp16"])}
    elif kind == "layer":
        layout = rng.choice(["channels_first", "channels_last"])
        dim, heads = rng.choice([(128, 2), (128, 8), (192, 4), (256, 4), (256, 8), (256, 16), (512, 8), (512, 16)])
        T = _log_int(rng, 40, 1000)
        batch = _log_int(rng, 1, max(1, min(512, LAYER_ELEMENTS // (T * dim))))
        groups = rng.choice([1, 2, 4, 8]) if layout == "channels_first" else 1
        case = _layer("", layout, batch, T, dim, heads, _log_int(rng, 3, 33), groups, rng.random() < 0.6,
                      rng.choice(["autocast", "autocast", "fp16"]), rng.choice([1, 1, 1, 2]))
    else:
        train = rng.random() < 0.5
        frames = _log_int(rng, 100, 400)
        most = (128 if train else 512) * 300 // frames
        batch = _log_int(rng, min(most, 96) if train else 8, min(512, most))
        case = _model("", batch, frames, rng.choice([4, 8, 16]), rng.choice([5, 7, 9, 15, 27]), train)
    case.pop("name", None)
    return case


def prepare(case, seed):
    dev = torch.device("cuda", torch.cuda.current_device())
    g = torch.Generator(device=dev).manual_seed(seed)

    def randn(*shape, dtype=torch.float32, scale=1.0):
        return torch.randn(*shape, device=dev, generator=g).mul_(scale).to(dtype)

    def lengths(full):   # utterances between two thirds of the batch's longest and all of it
        return torch.randint(max(1, 2 * full // 3), full + 1, (case["batch"],), device=dev, generator=g, dtype=torch.int32)

    st = {"case": case}
    kind = case["kind"]
    if kind in ("op", "pair"):
        shape = (case["batch"] * case["heads"], case["T"], case["C"])
        dt = DTYPES[case["dtype"]]
        train = case.get("train", True)
        st["q"], st["k"], st["v"] = (randn(*shape, dtype=dt).requires_grad_(train) for _ in range(3))
        if train:
            st["d_o"] = randn(*shape, dtype=dt)
        st["rpb"] = None
        if kind == "pair" or case["bias"]:
            st["rpb"] = randn(1, case["heads"], 1, case["win"], scale=0.1).requires_grad_(train)
        if kind == "pair":
            left = case["win"] - 1 - case["win"] // 2
            st["left"], st["mask"] = left, padding_mask(case["T"], case["win"], left, case["dil"], device=dev)
            st["functions"] = getNA1dFunction(case["C"], case["dil"], dt)
        else:
            st["valid_len"] = lengths(case["T"]) if case["padded"] else None
            st["drop_seed"] = 1000003 * seed + 17
    elif kind == "layer":
        torch.manual_seed(seed)
        with dev:
            m = NAttention(case["T"], case["dim"], case["heads"], case["win"], case["dil"], case["groups"], layout=case["layout"])
        dt = torch.float16 if case["dtype"] == "fp16" else torch.bfloat16
        st["layer"] = (m.to(dt) if case["dtype"] == "fp16" else m).train(case["train"])
        B, T, D = case["batch"], case["T"], case["dim"]
        shape = (B, D, T) if case["layout"] == "channels_first" else (B, T, D)
        st["x"] = randn(*shape, dtype=dt).requires_grad_(case["train"])
        if case["train"]:
            st["d_y"] = randn(*shape, dtype=dt)
        else:
            st["padding"] = T - lengths(T)
    else:
        torch.manual_seed(seed)
        with dev:
            m = PCFNATExtractor(frames=case["frames"], heads=case["heads"], win=case["win"])
        st["model"] = m.train(case["train"])
        st["fbank"] = randn(case["batch"], FEAT, case["frames"])
        if case["train"]:
            st["labels"] = torch.randint(0, CLASSES, (case["batch"],), device=dev, generator=g)
            st["grads"] = flat_gradient_buffer(m.parameters())
        else:
            st["padding"] = case["frames"] - lengths(case["frames"])
    return st


def run(st):
    case = st["case"]
    return {"op": _run_op, "pair": _run_pair, "layer": _run_layer, "model": _run_model}[case["kind"]](case, st)


def _run_op(case, st):
    args = (st["q"], st["k"], st["v"], case["win"], case["left"], case["dil"], case["C"] ** -0.5, st["rpb"], st["valid_len"],
            case["heads"])
    if not case["train"]:
        with torch.no_grad():
            return na1d_fused(*args)
    o = na1d_fused(*args, drop_p=case["drop"], seed=st["drop_seed"]) if case["drop"] else na1d_fused(*args)
    leaves = [st["q"], st["k"], st["v"]] + ([st["rpb"]] if case["bias"] else [])
    return (o.detach(),) + torch.autograd.grad(o, leaves, st["d_o"])


def _run_pair(case, st):
    QK, AV = st["functions"]
    N, T, win = case["batch"] * case["heads"], case["T"], case["win"]
    attn = QK.apply(st["q"] * case["C"] ** -0.5, st["k"], win, st["left"], case["dil"])
    attn = attn.view(case["batch"], case["heads"], T, win) + st["rpb"]
    attn = (attn + st["mask"]).view(N, T, win).softmax(dim=-1)
    o = AV.apply(attn, st["v"], win, st["left"], case["dil"])
    return (o.detach(),) + torch.autograd.grad(o, (st["q"], st["k"], st["v"], st["rpb"]), st["d_o"])


def _run_layer(case, st):
    m = st["layer"]
    with torch.set_grad_enabled(case["train"]), torch.autocast("cuda", dtype=torch.bfloat16, enabled=case["dtype"] == "autocast"):
        y = m(st["x"], None if case["train"] else st["padding"])
    if not case["train"]:
        return y
    return (y.detach(),) + torch.autograd.grad(y, [st["x"]] + list(m.parameters()), st["d_y"])


def _run_model(case, st):
    m = st["model"]
    if not case["train"]:
        with torch.no_grad(), torch.autocast("cuda", dtype=torch.bfloat16):
            return m.embedding(st["fbank"], st["padding"])
    st["grads"].zero_()
    with torch.autocast("cuda", dtype=torch.bfloat16):
        loss = m(st["fbank"], st["labels"])
    loss.backward()
    return loss.detach(), st["grads"]


def _op_work(rows, C, win, train):
    """Forward: q, k, v in, o out. Backward (a pass of its own: its input depends on the forward's output): q, k, v, d_o in,
    three gradients out, and the row statistics handed from one to the other."""
    return ((22 * C + 8 if train else 8 * C) * rows, (14 if train else 4) * rows * win * C)


def work(case):
    kind = case["kind"]
    if kind == "op":
        b, f = _op_work(case["batch"] * case["heads"] * case["T"], case["C"], case["win"], case["train"])
    elif kind == "pair":
        # the fp32 band goes through memory between the operators: QK, two additions, softmax, AV and their backwards
        rows = case["batch"] * case["heads"] * case["T"]
        b, f = rows * (32 * case["C"] + 60 * case["win"]), 14 * rows * case["win"] * case["C"]
    elif kind == "layer":
        tokens, D = case["batch"] * case["T"], case["dim"]
        ob, of = _op_work(tokens * case["heads"], D // case["heads"], case["win"], case["train"])
        # input in and output out, the projected 3D channels and the merged heads between the three parts; weights
        proj_b, proj_f = tokens * D * 2 * (1 + 3 + 1 + 1), 8 * tokens * D * D // (1 if case["layout"] == "channels_last" else case["groups"])
        b, f = ob + proj_b * (3 if case["train"] else 1) + 16 * D * D, of + proj_f * (3 if case["train"] else 1)
    else:
        B, T = case["batch"], case["frames"]
        f = B * model_flops_per_utterance(frames=T, win=case["win"]) / (1 if case["train"] else 3)
        # features, weights (and their gradients); per block the residual stream in and out twice, the 3-fold projection, the
        # merged heads and the 4-fold hidden layer in and out, all 16-bit, three times over with the backward pass
        block = B * T * 256 * 2 * (4 + 6 + 2 + 8)
        b = B * FEAT * T * 4 + 4 * 22.5e6 * (2 if case["train"] else 1) + 24 * block * (3 if case["train"] else 1)
    return {"bytes": float(b), "flops": float(f)}


def tolerance(case):
    """About four times the distance from the same computation in 64 bits, measured over these ranges (2-norm / largest
    element): operator and layer gradients 2.4e-3 / 2.6e-2 (bf16) and 3.0e-4 / 3.7e-3 (fp16), whole layer 4.5e-3 / 2.7e-2 (bf16) and
    4.6e-4 / 2.7e-3 (fp16), embeddings 4.8e-3 / 1.8e-2. The network's gradient passes through 24 blocks in bf16: 1.5e-2, and
    its largest element, in the few class rows that a batch touches, differs by the order of the gradient's root mean square."""
    kind = case["kind"]
    if kind == "model":
        return {"rel": 0.03, "max": 0.99} if case["train"] else {"rel": 0.018, "max": 0.07}
    if kind == "layer":
        return {"rel": 0.002, "max": 0.012} if case["dtype"] == "fp16" else {"rel": 0.018, "max": 0.1}
    return {"rel": 0.0012, "max": 0.015} if case["dtype"] == "fp16" else {"rel": 0.01, "max": 0.1}


def _exact_attention(q, k, v, win, left, dil, scale, bias, valid):
    """softmax(scale q.k + bias + mask) . v over each token's window; q, k, v (batch, heads, T, C), bias (heads, win) or None,
    valid (batch,) tokens or None. A neighbour outside the sequence is a zero row under the mask's -100."""
    T = q.shape[2]
    lo, hi = left * dil, (win - 1 - left) * dil
    kp, vp = F.pad(k, (0, 0, lo, hi)), F.pad(v, (0, 0, lo, hi))
    t = torch.arange(T, device=q.device)
    n = torch.full((q.shape[0], 1), T, device=q.device) if valid is None else valid.long().view(-1, 1)
    logits = []
    for kk in range(win):
        j = t + (kk - left) * dil
        off = ((j < 0) | (j >= n) | (t >= n)).to(q.dtype).mul(-100.0)                                # (batch, T)
        x = (q * kp[:, :, kk * dil:kk * dil + T]).sum(-1) * scale + off[:, None]
        logits.append(x if bias is None else x + bias[:, kk].view(1, -1, 1))
    p = torch.softmax(torch.stack(logits, -1), -1)
    o = torch.zeros_like(q)
    for kk in range(win):
        o = o + p[..., kk, None] * vp[:, :, kk * dil:kk * dil + T]
    return o


def _exact_layer(x, w, layout, heads, groups, win, left, dil, scale, valid):
    """The attention layer on x with its parameters w[...]: projection, heads, attention, merge, projection."""
    if layout == "channels_first":
        B, D, T = x.shape
        y = F.conv1d(x, w["qkv.weight"], w["qkv.bias"], groups=groups)
        y = y.view(B, D // groups, groups, 3, T).transpose(1, 2).reshape(B, heads, D // heads, 3, T).permute(3, 0, 1, 4, 2)
    else:
        B, T, D = x.shape
        y = F.linear(x, w["qkv.weight"], w["qkv.bias"]).view(B, T, 3, heads, D // heads).permute(2, 0, 3, 1, 4)
    o = _exact_attention(y[0], y[1], y[2], win, left, dil, scale, w["relative_position_bias"].view(heads, win), valid)
    if layout == "channels_first":
        return F.conv1d(o.transpose(2, 3).reshape(B, D, T), w["proj.weight"], w["proj.bias"], groups=groups)
    return F.linear(o.transpose(1, 2).reshape(B, T, D), w["proj.weight"], w["proj.bias"])


def _exact_model(case, m, w, fbank, labels, valid):
    def norm(x, name):
        return F.layer_norm(x, x.shape[-1:], w[name + ".weight"], w[name + ".bias"], 1e-5)

    def linear(x, name):
        return F.linear(x, w[name + ".weight"], w[name + ".bias"])

    win, left = case["win"], case["win"] - 1 - case["win"] // 2
    x = F.conv1d(fbank, w["front.weight"], w["front.bias"], padding=2).transpose(1, 2)
    feats, outs, stages = [x], [], len(m.stages)
    for s in range(stages):
        for i in range(len(m.stages[s])):
            name = "stages.%d.%d." % (s, i)
            attn = {n[len(name) + 5:]: p for n, p in w.items() if n.startswith(name + "attn.")}
            x = x + _exact_layer(norm(x, name + "norm1"), attn, "channels_last", case["heads"], 1, win, left, 1,
                                 (x.shape[-1] // case["heads"]) ** -0.5, valid)
            x = x + linear(F.gelu(linear(norm(x, name + "norm2"), name + "fc1")), name + "fc2")
        outs.append(x)
        feats.append(x)
        if s + 1 < stages:
            x = linear(torch.cat(feats, -1), "fuse.%d" % s)
    y = torch.cat(outs, -1)
    a = torch.softmax(linear(torch.tanh(linear(y, "pool.a")), "pool.b"), 1)
    mu = (a * y).sum(1)
    y = torch.cat([mu, ((a * y * y).sum(1) - mu * mu).clamp_min(1e-5).sqrt()], 1)
    stats = (None, None) if case["train"] else (m.bn.running_mean.double(), m.bn.running_var.double())
    y = linear(F.batch_norm(y, stats[0], stats[1], w["bn.weight"], w["bn.bias"], case["train"], 0.0, 1e-5), "embed")
    if labels is None:
        return y
    cos = F.linear(F.normalize(y), F.normalize(w["loss.weight"])).clamp(-1 + 1e-7, 1 - 1e-7)
    target = torch.cos(torch.acos(cos.gather(1, labels[:, None])) + 0.2)
    return F.cross_entropy(cos.scatter(1, labels[:, None], target) * 30.0, labels)


def exact(case, seed):
    """What ``run`` returns, in 64 bits by plain torch on the same inputs. Not for attention dropout (its mask is the
    operator's own) and not for the network's larger batches, whose activations do not fit in 64 bits."""
    kind = case["kind"]
    if case.get("drop") or (kind == "model" and case["batch"] * case["frames"] > (9600 if case["train"] else 80000)):
        return None
    st = prepare(case, seed)
    train = case.get("train", True)
    with torch.set_grad_enabled(train):
        if kind in ("op", "pair"):
            B, H, T, C, win = (case[n] for n in ("batch", "heads", "T", "C", "win"))
            left = st["left"] if kind == "pair" else case["left"]
            q, k, v = (st[n].detach().double().requires_grad_(train) for n in "qkv")
            r = None if st["rpb"] is None else st["rpb"].detach().double().requires_grad_(train)
            o = _exact_attention(*(x.view(B, H, T, C) for x in (q, k, v)), win, left, case["dil"], C ** -0.5,
                                 None if r is None else r.view(H, win), st.get("valid_len")).reshape(B * H, T, C)
            if not train:
                return o
            return (o.detach(),) + torch.autograd.grad(o, [q, k, v] + ([] if r is None else [r]), st["d_o"].double())
        m = st["layer" if kind == "layer" else "model"]
        w = {n: p.detach().double().requires_grad_(train) for n, p in m.named_parameters()}
        valid = (case["T"] if kind == "layer" else case["frames"]) - st["padding"] if "padding" in st else None
        if kind == "layer":
            x = st["x"].detach().double().requires_grad_(train)
            y = _exact_layer(x, w, case["layout"], case["heads"], case["groups"], case["win"], case["win"] - 1 - case["win"] // 2,
                             case["dil"], (case["dim"] // case["heads"]) ** -0.5, valid)
            return (y.detach(),) + torch.autograd.grad(y, [x] + list(w.values()), st["d_y"].double()) if train else y
        out = _exact_model(case, m, w, st["fbank"].double(), st.get("labels"), valid)
        if not train:
            return out
        return out.detach(), torch.cat([g.reshape(-1) for g in torch.autograd.grad(out, list(w.values()))])
