"""Reference (CPU) paths of the fused functional ops agree with their unfused compositions."""
import ctypes
import os

import pytest
import torch

from libai_b200 import ops
from libai_b200.ops import functional as OF
from libai_b200.ops import so_path


def test_linear_bias_residual_and_mlp_residual_reference_paths():
    torch.manual_seed(0)
    x, w, b, r = torch.randn(6, 16), torch.randn(8, 16), torch.randn(8), torch.randn(6, 8)
    assert torch.allclose(OF.linear_bias_residual(x, w, b, r), x @ w.t() + b + r, atol=1e-5)
    assert torch.allclose(OF.linear_bias_residual(x, w, None, None), x @ w.t(), atol=1e-5)
    w1, b1, w2, b2, res = torch.randn(12, 16), torch.randn(12), torch.randn(16, 12), torch.randn(16), torch.randn(6, 16)
    want = torch.nn.functional.gelu(x @ w1.t() + b1) @ w2.t() + b2 + res
    assert torch.allclose(OF.mlp(x, w1, b1, w2, "gelu", b2, res), want, atol=1e-4)
    assert torch.allclose(OF.mlp(x, w1, b1, w2, "gelu"), want - b2 - res, atol=1e-4)


def test_layer_norm_with_skip_reference_path():
    torch.manual_seed(0)
    x = torch.randn(4, 10, requires_grad=True)
    g, b = torch.randn(10), torch.randn(10)
    ln, skip = OF.layer_norm_with_skip(x, g, b)
    assert skip is x
    assert torch.allclose(ln, torch.nn.functional.layer_norm(x, (10,), g, b, 1e-5), atol=1e-5)
    (ln.sum() + (skip * 2).sum()).backward()
    assert x.grad is not None and torch.isfinite(x.grad).all()


@pytest.mark.parametrize("moved", range(5))
def test_attention_kernels_are_not_given_tensors_of_another_device(moved, monkeypatch):
    """A cache, or keys and values, held on another device than the queries: the kernels are not taken (no launch here: the support
    checks are asked, the extension is a stand-in that records a call)."""

    class Reached(Exception):
        pass

    class Ext:
        def __getattr__(self, name):
            raise Reached(name)

    monkeypatch.setattr(OF, "use_native", lambda *t: True)
    monkeypatch.setattr(OF, "load_ext", lambda *a, **k: Ext())
    at = lambda i, *shape: torch.zeros(*shape, dtype=torch.bfloat16, device="meta" if i == moved else "cpu")
    new, past = (2, 3, 1, 32), (2, 3, 7, 32)
    with pytest.raises(Reached):
        OF.attention_cached(*(at(-1, *s) for s in (new, new, new, past, past)), scale=0.1)
    assert OF.attention_cached(*(at(i, *s) for i, s in enumerate((new, new, new, past, past))), scale=0.1) is None
    if moved < 3:
        assert OF._split_supported(*(at(-1, *past) for _ in range(3)), 0.1, False, None)
        assert not OF._split_supported(*(at(i, *past) for i in range(3)), 0.1, False, None)
    if moved < 2:
        assert OF.attention_packed("q_kv", (at(0, 2, 7, 3, 32), at(1, 2, 9, 3, 64)), causal=False, scale=0.1) is None


@pytest.mark.skipif(torch.cuda.is_available() or not os.path.exists(so_path()), reason="host side of the C entry only: no launch may follow")
def test_norm_backward_never_drops_the_residual_gradient():
    """A gradient of the residual path is added by the kernel or refused (-3), whichever of the tensors is not on 16 bytes; the pointers
    are only looked at."""
    lib = ctypes.CDLL(so_path())
    p = lambda at: ctypes.c_void_p(at)
    for odd in range(5):
        gy, x, gamma, gx, gadd = (p(0x10000 * (i + 1) + (8 if i == odd else 0)) for i in range(5))
        assert lib.lb_norm_bwd(gy, x, gamma, p(0), p(0x90000), gx, p(0xa0000), p(0), p(0xb0000), 4, 512, 1, 0, 0, 0, gadd, p(0)) == -3
        assert lib.lb_norm_bwd_supports_gadd(512, 0, gy, x, gamma, gx, gadd) == 0
    aligned = [p(0x10000 * (i + 1)) for i in range(5)]
    assert lib.lb_norm_bwd_supports_gadd(512, 0, *aligned) == 1


@pytest.mark.skipif(torch.cuda.is_available() or not os.path.exists(so_path()), reason="host side of the C entry only: no launch may follow")
@pytest.mark.parametrize("width,layout,epi", [(-64, 0, 0), (-96, 2, 2), (100, 0, 0), (320, 1, 0), (-128, 0, 1), (-192, 0, 2), (-128, 1, 1), (-192, 1, 2), (-128, 2, 0), (-192, 2, 1)])
def test_gemm_refuses_forced_widths_without_a_kernel(width, layout, epi):
    """-1 before a tensor map is made (-2 where that has no driver): a 256-wide kernel on boxes of another width would wait for bytes that nobody sends."""
    lib, p = ctypes.CDLL(so_path()), ctypes.c_void_p
    call = lambda w, lay, e: lib.lb_gemm_bf16(p(0x10000), p(0x20000), p(0x30000), 512, 512, 512, 512, 512, 512, lay, e, p(0), 0, p(0), w, 1, p(0))
    assert call(width, layout, epi) == -1
    assert call(-256, layout, epi) == call(256, layout, epi) == call(64, layout, epi) == -2


@pytest.mark.skipif(torch.cuda.is_available() or not os.path.exists(so_path()), reason="host side of the C entry only")
@pytest.mark.parametrize("m,n,k,few", [(8, 1024, 4096, 1), (200, 1024, 4096, 1), (128, 4096, 1024, 1), (2048, 4096, 1024, 0), (8192, 1024, 1024, 0)])
def test_rule_of_few_rows_answers_without_a_device(m, n, k, few):
    nt, ranks = ctypes.c_int(0), ctypes.c_int(0)
    assert ctypes.CDLL(so_path()).lb_gemm_small_rule(m, n, k, ctypes.byref(nt), ctypes.byref(ranks)) == few


@pytest.mark.skipif(torch.cuda.is_available() or not os.path.exists(so_path()), reason="host side of the C entry only")
@pytest.mark.parametrize("h", [8, 512, 1024, 1280, 4096, 8192])
def test_workspace_of_norm_backward(h):
    """One row per block, none for no rows."""
    rows = ctypes.CDLL(so_path()).lb_norm_bwd_workspace_rows
    assert rows(0, h) == 0 and rows(1, h) == 1
    assert all(0 < rows(n, h) <= min(n, 3 * 148) for n in (2, 5, 148, 593, 1777, 8192, 100000))


def test_implementation_switch_follows_the_environment(monkeypatch):
    monkeypatch.delenv("LIBAI_B200_IMPL", raising=False)
    assert ops.impl() == "native"
    monkeypatch.setenv("LIBAI_B200_IMPL", "ref")
    assert ops.impl() == "ref"
    monkeypatch.setattr(os, "environ", {"LIBAI_B200_IMPL": "other"})       # the whole mapping replaced
    assert ops.impl() == "other"
    monkeypatch.setattr(os, "environ", {})
    assert ops.impl() == "native"
