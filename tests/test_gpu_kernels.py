"""GPU tier: single kernels of the training path at the sizes where a tile, a remainder or a wait can go wrong, against plain PyTorch."""
import math

import pytest
import torch

from libai_b200.ops import functional as OF

pytestmark = pytest.mark.gpu
BF16 = torch.bfloat16


def _rand(shape, seed=0, std=1.0, dtype=BF16):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.empty(shape, device="cuda", dtype=torch.float32).normal_(0.0, std, generator=g).to(dtype)


def _attend64(q, k, v, scale, keep=None):
    """float64 softmax attention on ``[b, a, s, d]``; where ``keep`` is false the score is -10000."""
    s = q.double() @ k.double().transpose(-1, -2) * scale
    if keep is not None:
        s = torch.where(keep, s, torch.full_like(s, -10000.0))
    return torch.softmax(s, -1) @ v.double()


@pytest.mark.parametrize("dim", [64, 128])
@pytest.mark.parametrize("causal", [True, False])
def test_attention_rows_do_not_depend_on_timing(dim, causal):
    """Many CTAs on every SM: no row of any repetition may differ, and every row is right (probabilities of one key block must
    not be overwritten while the tensor core still reads them)."""
    b, s, a = 4, 1024, 16
    qkv = _rand((b, s, a, 3 * dim))
    q, k, v = (t.permute(0, 2, 1, 3) for t in qkv.split(dim, -1))
    keep = torch.ones(s, s, dtype=torch.bool, device="cuda").tril() if causal else None
    first = OF.attention_qkvpacked(qkv, causal=causal, scale=dim ** -0.5)
    want = torch.cat([_attend64(q[i:i + 1], k[i:i + 1], v[i:i + 1], dim ** -0.5, keep) for i in range(b)]).permute(0, 2, 1, 3)
    row = (first.double() - want).norm(dim=-1) / want.norm(dim=-1)
    # probabilities and results are rounded to bf16 (2^-9 each); a long row averages them, a short one has few of them
    assert float(row.max()) < 4 * 2.0 ** -8
    for _ in range(5):
        assert torch.equal(OF.attention_qkvpacked(qkv, causal=causal, scale=dim ** -0.5), first)
