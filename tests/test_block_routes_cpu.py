"""Which blocks the one-node route takes (host-only decisions), and that every other block runs its own forward."""
import os
import subprocess
import sys

import torch
import torch.nn as nn

from pcf_nat_b200 import block
from pcf_nat_b200.model import NABlock, PCFNATExtractor


class _Scaled(NABlock):
    def forward(self, x, padding=None):
        return x + 0.5 * (super().forward(x, padding) - x)


def _taken(cls=NABlock, change=lambda b: b):
    blk = change(cls(40, 64, 2, 7, 4, "fused"))
    return block._block_parameters(blk, torch.zeros(2, 40, 64)) is not None


def test_only_the_plain_block_is_taken():
    from torch.distributed.algorithms._checkpoint.checkpoint_wrapper import checkpoint_wrapper
    assert _taken()
    assert not _taken(_Scaled)
    assert not _taken(change=checkpoint_wrapper)
    assert not _taken(change=lambda b: nn.Sequential(b))


def test_blocks_without_the_attributes_of_the_plain_one_run():
    class Half(nn.Module):
        def forward(self, x, padding=None):
            return 0.5 * x

    m = PCFNATExtractor(frames=30, feat=8, dim=32, heads=2, win=7, stages=2, blocks=1, emb=16, classes=10).eval()
    for s in m.stages:
        s[0] = Half()
    with torch.no_grad():
        assert m.embedding(torch.randn(2, 8, 30), torch.tensor([0, 3])).shape == (2, 16)


def test_dropout_follows_the_flag_of_its_own_module():
    def set_(attn=0.0, proj=0.0, training=False, proj_training=False):
        def change(b):
            b.train(training)
            b.attn.attn_drop.p, b.attn.proj_drop.p = attn, proj
            b.attn.proj_drop.train(proj_training)
            return b
        return change

    assert _taken(change=set_(attn=0.1, proj=0.1))                      # evaluation: neither is applied
    assert not _taken(change=set_(proj=0.1, proj_training=True))        # evaluation with the dropout modules in training mode
    assert not _taken(change=set_(attn=0.1, training=True))             # the layer's own flag decides about attention dropout
    assert not _taken(change=set_(proj=0.1, training=True, proj_training=True))
    assert _taken(change=set_(proj=0.1, training=True))


WITHOUT_NODES = """
import sys, warnings
sys.modules["pcf_nat_b200._na1d_torch"] = None        # as if it were not built
with warnings.catch_warnings(record=True) as seen:
    warnings.simplefilter("always")
    import pcf_nat_b200
    from pcf_nat_b200 import ops
assert any("_na1d_torch" in str(w.message) for w in seen)
assert not ops.native.eager_mode() and ops.native.fused(1, 2) is None
"""


def test_package_imports_without_the_extension_of_nodes():
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    subprocess.run([sys.executable, "-c", WITHOUT_NODES], cwd=root, check=True)


def test_pooling_hands_its_projection_the_rows_as_they_came():
    from pcf_nat_b200.model import AttentiveStatsPool
    torch.manual_seed(0)
    pool = AttentiveStatsPool(16)
    x, shapes = torch.randn(3, 16, 20).transpose(1, 2), []          # not contiguous
    want = pool(x.contiguous())
    assert torch.allclose(pool(x), want, rtol=1e-5, atol=1e-6)
    pool.a.register_forward_hook(lambda m, i, o: shapes.append(i[0].shape))
    assert torch.allclose(pool(x), want, rtol=1e-5, atol=1e-6) and shapes == [x.shape]
