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


@pytest.mark.parametrize("rms", [False, True])
@pytest.mark.parametrize("rows,h", [(1, 8), (3, 192), (257, 384), (2048, 768), (130, 1000), (515, 1024), (4, 1032), (300, 1280), (37, 2048),
                                    (450, 4096), (33, 6152), (5, 8192), (3, 8200), (9, 99)])
def test_norm_kernels_at_their_edges(rows, h, rms):
    """Rows of a warp (up to 1024 columns), of a block (up to 8192) and of the generic kernel, forward, backward, with the gradient of a
    residual path, into new tensors and into fp32 gradients."""
    x, gy, skip = _rand((rows, h), 1), _rand((rows, h), 2), _rand((rows, h), 3)
    w, b = _rand((h,), 4), None if rms else _rand((h,), 5)
    x64, w64 = x.double().requires_grad_(True), w.double().requires_grad_(True)
    b64 = None if rms else b.double().requires_grad_(True)
    d = x64 if rms else x64 - x64.mean(-1, keepdim=True)
    y64 = d * torch.rsqrt(d.square().mean(-1, keepdim=True) + 1e-5) * w64
    y64 = y64 if rms else y64 + b64
    y64.backward(gy.double())
    ext = OF.load_ext()
    y, mean, rstd = ext.norm_fwd(x, w, b, 1e-5, rms)
    close = lambda got, want, tol: float((got.double() - want).norm() / want.norm().clamp_min(1e-30)) < tol
    assert close(y, y64, 2.0 ** -8)                              # one rounding to bf16
    for acc in (False, True):
        gw = torch.ones(h, device="cuda") if acc else None
        gb = torch.ones(h, device="cuda") if acc and not rms else None
        gx, dw, db = ext.norm_bwd(gy, x, w, mean, rstd, rms, not rms, gw, gb, skip)
        dw, db = (gw - 1, None if rms else gb - 1) if acc else (dw, db)
        assert close(gx, x64.grad + skip.double(), 2.0 ** -7)    # bf16, and once more where the residual gradient is added outside
        assert close(dw, w64.grad, 1e-5) and (rms or close(db, b64.grad, 1e-5))


@pytest.mark.parametrize("b,s,a,d,off", [(1, 1, 1, 16, 0), (2, 37, 3, 128, 5), (1, 2100, 4, 64, 0), (3, 9, 5, 48, 1), (2, 7, 2, 24, 3), (1, 5, 32, 256, 0)])
def test_rotary_on_the_packed_projection(b, s, a, d, off):
    qkv, g = _rand((b, s, a, 3 * d), 1), _rand((b, s, a, 3 * d), 2)
    ang = torch.outer(torch.arange(s + off, device="cuda").float(), 1.0 / 10000 ** (torch.arange(0, d, 2, device="cuda") / d))
    cos, sin = torch.cat([ang, ang], -1).cos().contiguous(), torch.cat([ang, ang], -1).sin().contiguous()
    x = qkv.clone().requires_grad_(True)
    y = OF.apply_rotary_qkv(x, cos, sin, off)
    x64 = qkv.double().requires_grad_(True)
    c, n = cos[off:off + s, None].double(), sin[off:off + s, None].double()
    q, k, v = x64.split(d, -1)
    y64 = torch.cat([q * c + OF.rotate_half(q) * n, k * c + OF.rotate_half(k) * n, v], -1)
    y.backward(g.clone())
    y64.backward(g.double())
    assert float((y.double() - y64).norm() / y64.norm()) < 2.0 ** -8
    assert float((x.grad.double() - x64.grad).norm() / x64.grad.norm()) < 2.0 ** -8
