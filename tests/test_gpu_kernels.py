"""GPU tier: single kernels of the training path at the sizes where a tile, a remainder or a wait can go wrong, against plain PyTorch."""
import ctypes
import gc
import math

import pytest
import torch
from torch._subclasses.fake_tensor import FakeTensorMode

from libai_b200.ops import functional as OF
from libai_b200.ops import load_ext, so_path
from libai_b200.ops.gated_mlp import gated_mlp

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


@pytest.mark.parametrize("lens", [False, True])
@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("dim", [64, 128])
@pytest.mark.parametrize("b,s,a,packed", [(1, 8, 1, True), (2, 64, 3, False), (1, 65, 2, True), (2, 129, 200, True), (1, 192, 40, False), (3, 257, 70, True),
                                          (2, 385, 80, True), (1, 1096, 33, False), (90, 200, 8, True), (1, 2049, 16, True)])
def test_attention_forward_two_tiles_per_block(b, s, a, packed, dim, causal, lens):
    """One unit of 64 keys and many, one query tile or two per work item, an odd number of tiles, last units of every width, fewer and
    more work items than SMs: result and log-sum-exp against float64, the same bits again."""
    if packed:
        q, k, v = (t.permute(0, 2, 1, 3) for t in _rand((b, s, a, 3 * dim), 1).split(dim, -1))
    else:
        q, k, v = (_rand((b, a, s, dim), 1 + i) for i in range(3))
    n = torch.tensor([max(1, s - 29 * i * i) for i in range(b)], dtype=torch.int32, device="cuda") if lens else None
    o, lse, _ = load_ext().attn_fwd(q, k, v, causal, dim ** -0.5, n, None, None, 0.0, 0)
    assert o.transpose(1, 2).is_contiguous()
    for i in range(0, b, max(1, b // 3)):
        z = q[i].double() @ k[i].double().transpose(-1, -2) * dim ** -0.5
        keep = torch.ones(s, s, dtype=torch.bool, device="cuda")
        keep = keep.tril() if causal else keep
        if lens:
            keep = keep & (torch.arange(s, device="cuda")[None] < n[i])
        z = z.masked_fill(~keep, -math.inf)
        prob = torch.softmax(z, -1)
        want = prob @ v[i].double()
        # a probability is rounded to bf16 (8 bits: by at most 2^-8 of it, so by 2^-8 of the sum of |p v|), the result once more; 2^-13 for all fp32
        assert bool(((o[i].double() - want).abs() <= (2.0 ** -8 + 2.0 ** -13) * (prob @ v[i].double().abs() + want.abs())).all())
        # scores are fp32 sums of `dim` products
        assert float((lse[i].double() - torch.logsumexp(z, -1)).abs().max()) < 2.0 ** -24 * dim * max(1.0, float(z[keep.expand_as(z)].abs().max()))
    for _ in range(2):
        o2, lse2, _ = load_ext().attn_fwd(q, k, v, causal, dim ** -0.5, n, None, None, 0.0, 0)
        assert torch.equal(o, o2) and torch.equal(lse, lse2)


@pytest.mark.parametrize("rms", [False, True])
@pytest.mark.parametrize("rows,h", [(1, 8), (3, 192), (257, 384), (2048, 768), (130, 1000), (515, 1024), (4, 1032), (300, 1280), (37, 2048),
                                    (450, 4096), (33, 6152), (5, 8192), (3, 8200), (9, 99),
                                    (296, 1280), (297, 1280), (1536, 1280), (600, 1536), (1535, 2048), (2048, 2048), (2100, 2560), (2048, 1792), (2048, 2304), (1024, 2048), (888, 2048)])
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


@pytest.mark.parametrize("rms", [False, True])
@pytest.mark.parametrize("rows,h", [(2048, 4096), (300, 1280), (700, 8192)])
def test_norm_weight_gradients_of_wide_rows_repeat(rows, h, rms):
    """Added to fp32 gradients by many blocks: the same bits every time."""
    x, gy, w = _rand((rows, h), 1), _rand((rows, h), 2), _rand((h,), 4)
    ext = OF.load_ext()
    _, mean, rstd = ext.norm_fwd(x, w, None if rms else w, 1e-5, rms)
    runs = []
    for _ in range(6):
        gw, gb = torch.ones(h, device="cuda"), None if rms else torch.ones(h, device="cuda")
        ext.norm_bwd(gy, x, w, mean, rstd, rms, not rms, gw, gb, None)
        runs.append(gw if rms else torch.cat([gw, gb]))
    assert all(torch.equal(r, runs[0]) for r in runs)


@pytest.mark.parametrize("b,s,a,d,off", [(1, 1, 1, 16, 0), (2, 37, 3, 128, 5), (1, 2100, 4, 64, 0), (3, 9, 5, 48, 1), (2, 7, 2, 24, 3), (1, 5, 32, 256, 0),
                                         (1, 1, 64, 128, 9), (4, 1, 37, 128, 0), (1, 700, 12, 64, 0)])
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


def _split_mask(kind, b, a, sq, sk):
    g = torch.Generator(device="cuda").manual_seed(11)
    on = torch.rand(b, 1, sq, sk, device="cuda", generator=g) < 0.6
    on[:, :, sq // 2] = False                                       # a query that sees no key: uniform over all of them
    if kind == "bool":
        return on
    if kind == "keys_int64":
        return on[:, :, :1].long() * 3
    if kind == "float_2d":
        return torch.where(on[0, 0], 0.5, -0.0)                     # a negative zero masks
    if kind == "heads_strided":
        heads = torch.rand(sk, a, sq, device="cuda", generator=g) < 0.5
        return heads.to(torch.int8).permute(1, 2, 0)[None]
    return None


@pytest.mark.parametrize("mask", ["none", "causal", "bool", "keys_int64", "float_2d", "heads_strided"])
@pytest.mark.parametrize("b,sq,sk,a,d", [(1, 1, 1, 1, 8), (2, 128, 136, 3, 64), (2, 129, 257, 2, 48), (1, 300, 300, 2, 24), (3, 17, 512, 2, 32),
                                         (2, 200, 130, 1, 40), (1, 127, 385, 2, 56), (1, 1, 700, 5, 16)])
def test_attention_with_32_bit_probabilities(b, sq, sk, a, d, mask):
    """Head dims up to 64, lengths around the 128-wide tiles, masks of every type and broadcast; forward and backward are as close to
    64-bit arithmetic as the unfused fp32 form that these calls took before."""
    causal = mask == "causal"
    if causal and sk < sq:
        pytest.skip("more queries than keys under a causal mask: unfused form")
    m = _split_mask(mask, b, a, sq, sk)
    q, k, v, go = _rand((b, a, sq, d), 1), _rand((b, sk, a, d), 2).permute(0, 2, 1, 3), _rand((b, a, sk, d), 3), _rand((b, a, sq, d), 4)
    keep = torch.ones(sq, sk, dtype=torch.bool, device="cuda").tril(sk - sq) if causal else None if m is None else m.bool()
    got = []
    for fn in (lambda *t: OF.attention(*t, causal=causal, scale=0.3, mask=m),
               lambda *t: OF.attention_ref(*t, causal=causal, scale=0.3, mask=m),
               lambda *t: _attend64(*t, 0.3, keep)):
        ts = [t.detach().clone().requires_grad_(True) for t in (q, k, v)]
        before = OF.ops.launch_count()
        y = fn(*ts)
        if not got:
            assert OF.ops.launch_count() > before and OF._split_supported(q, k, v, 0.3, causal, m)
        y.backward(go.to(y.dtype))
        got.append([y] + [t.grad for t in ts])
        if len(got) == 2:
            q, k, v, go = (t.double() for t in (q, k, v, go))
    for new, old, want in zip(*got):
        err = [float((t.double() - want).norm()) for t in (new, old)]
        # both round once to bf16: the errors differ by chance only, and by the fp32 sums' order where the results cancel to nothing
        assert err[0] <= 1.3 * err[1] + 1e-5 * float(want.norm()) + 1e-6 * math.sqrt(want.numel()), err


@pytest.mark.parametrize("mask", ["none", "causal", "bool"])
@pytest.mark.parametrize("b,sq,sk,a,d,common", [(2, 512, 512, 4, 48, 20.0), (1, 700, 700, 4, 24, 20.0), (1, 128, 1100, 2, 64, 6.0)])
def test_attention_of_keys_and_values_with_a_common_part(b, sq, sk, a, d, common, mask):
    """Biases of the projections give all keys and all values of a head a common part, which dP - delta and the sum of dS·K cancel:
    probabilities and their gradients need their 24 bits there.  No output further from 64 bits than the unfused fp32 form's; what
    the order of fp32 sums leaves (2^-24 of dP, some hundred times the result of the cancellation) may add a tenth."""
    causal = mask == "causal"
    m = _split_mask(mask, b, a, sq, sk)
    keep = torch.ones(sq, sk, dtype=torch.bool, device="cuda").tril(sk - sq) if causal else None if m is None else m.bool()
    q, go = _rand((b, a, sq, d), 1), _rand((b, a, sq, d), 4)
    k, v = ((_rand((b, a, sk, d), i).float() + common * _rand((1, a, 1, d), i + 4).float()).to(BF16) for i in (2, 3))
    got = []
    for fn, to in ((OF.attention, BF16), (OF.attention_ref, BF16), (None, torch.float64)):
        ts = [t.to(to).requires_grad_(True) for t in (q, k, v)]
        y = _attend64(*ts, d ** -0.5, keep) if fn is None else fn(*ts, causal=causal, scale=d ** -0.5, mask=m)
        got.append([y, *torch.autograd.grad(y, ts, go.to(to))])
    for new, old, want in zip(*got):
        err = [float((t.double() - want).norm()) for t in (new, old)]
        assert err[0] <= 1.1 * err[1], err


@pytest.mark.parametrize("mask", ["none", "causal", "bool"])
@pytest.mark.parametrize("b,sq,sk,a,d", [(8, 512, 512, 8, 48), (4, 200, 1100, 4, 32), (2, 700, 700, 4, 64)])
def test_attention_gradients_of_many_key_blocks_repeat(b, sq, sk, a, d, mask):
    """Every query's gradient is added up over the key blocks in their order: the same bits every time."""
    causal = mask == "causal"
    m = torch.ones(1, 1, 1, sk, dtype=torch.bool, device="cuda") if d == 64 and mask == "none" else _split_mask(mask, b, a, sq, sk)
    q, k, v = (_rand((b, a, s, d), i).requires_grad_(True) for i, s in ((1, sq), (2, sk), (3, sk)))
    m = torch.ones(sq, sk, dtype=torch.bool, device="cuda").tril(sk - sq) if d == 64 and causal else m      # head dim 64 takes these kernels with a mask
    out, go = OF.attention(q, k, v, causal=causal and d != 64, scale=d ** -0.5, mask=m), _rand((b, a, sq, d), 4)
    first = torch.autograd.grad(out, (q, k, v), go, retain_graph=True)
    for _ in range(5):
        assert all(torch.equal(x, y) for x, y in zip(torch.autograd.grad(out, (q, k, v), go, retain_graph=True), first))


@pytest.mark.parametrize("layout", ["qkv", "q_kv"])
def test_attention_from_packed_projections(layout):
    b, s, sk, a, d = 2, 150, 150 if layout == "qkv" else 333, 3, 48
    keep = torch.rand(b, 1, s, sk, device="cuda") < 0.7
    ts = [_rand((b, s, a, 3 * d), 1)] if layout == "qkv" else [_rand((b, s, a, d), 1), _rand((b, sk, a, 2 * d), 2)]
    go, out = _rand((b, s, a, d), 3), []
    for packed in (True, False):
        xs = [t.clone().requires_grad_(True) for t in ts]
        if packed:
            y = OF.attention_packed(layout, tuple(xs), causal=False, scale=d ** -0.5, mask=keep)
        else:
            y = _attend64(*OF._split_views(layout, xs), d ** -0.5, keep).permute(0, 2, 1, 3)
        y.backward(go.to(y.dtype))
        out.append([y] + [x.grad for x in xs])
    for got, want in zip(*out):
        assert float((got.double() - want.double()).norm() / want.double().norm()) < 2.0 ** -7


def test_attention_gradients_can_be_differentiated_again():
    q, k, v = (_rand((1, 2, 20, 24), i).requires_grad_(True) for i in range(3))
    (g,) = torch.autograd.grad(OF.attention(q, k, v, scale=0.2).float().square().sum(), q, create_graph=True)
    (h,) = torch.autograd.grad(g.float().square().sum(), k)
    ref = [t.detach().double().requires_grad_(True) for t in (q, k, v)]
    (g64,) = torch.autograd.grad(_attend64(*ref, 0.2).square().sum(), ref[0], create_graph=True)
    (h64,) = torch.autograd.grad(g64.square().sum(), ref[1])
    assert float((h.double() - h64).norm() / h64.norm()) < 0.05      # three bf16 roundings in a chain of products


@pytest.mark.parametrize("mask", [None, "bool", "int64"])
@pytest.mark.parametrize("b,a,past,d", [(1, 1, 1, 8), (8, 16, 511, 64), (2, 3, 63, 24), (3, 2, 1000, 128), (1, 4, 64, 48), (2, 1, 300, 256), (5, 7, 129, 16),
                                        (1, 2, 600, 8), (2, 1, 1030, 16)])
def test_attention_against_a_cache(b, a, past, d, mask):
    """One new token: context and grown caches, caches as strided views, with and without masked keys, every split over a cluster."""
    qkv = _rand((b, 1, a, 3 * d), 1)
    q, k, v = qkv.permute(0, 2, 1, 3).chunk(3, -1)
    kp, vp = _rand((b, past, a, d), 2).permute(0, 2, 1, 3), _rand((b, a, past, d), 3)
    m = None
    if mask is not None:
        m = torch.rand(b, 1, 1, past + 1, device="cuda") < 0.6
        m[0] = False                                                # no visible key at all: uniform
        m = m if mask == "bool" else m.long() * 2
    got = OF.attention_cached(q, k, v, kp, vp, scale=d ** -0.5, mask=m)
    key, value = torch.cat([kp, k], 2), torch.cat([vp, v], 2)
    assert torch.equal(got[1], key) and torch.equal(got[2], value)
    want = _attend64(q, key, value, d ** -0.5, None if m is None else m.bool()).permute(0, 2, 1, 3)
    old = OF.attention_ref(q, key, value, causal=False, scale=d ** -0.5, mask=m).permute(0, 2, 1, 3)
    err = [float((t.double() - want).norm()) for t in (got[0], old)]
    assert err[0] <= 1.3 * err[1] + 1e-5 * float(want.norm()), err   # both: fp32 throughout, one rounding to bf16


def test_cache_of_few_heads_and_a_very_long_past():
    """On both sides of the line between the one-kernel step and the concatenation."""
    for heads, past, d, one_kernel in ((1, 2000, 64, True), (1, 8900, 128, True), (1, 9100, 128, False), (2, 30000, 64, True), (2, 30000, 128, False), (3, 1000, 256, True), (4, 60000, 128, True)):
        q, k, v = (_rand((1, heads, 1, d), i) for i in range(3))
        kp, vp = _rand((1, heads, past, d), 4), _rand((1, heads, past, d), 5)
        got = OF.attention_cached(q, k, v, kp, vp, scale=d ** -0.5)
        assert (got is not None) == one_kernel
        if one_kernel:
            want = _attend64(q, torch.cat([kp, k], 2), torch.cat([vp, v], 2), d ** -0.5).permute(0, 2, 1, 3)
            assert float((got[0].double() - want).norm() / want.norm()) < 2.0 ** -8


@pytest.mark.parametrize("m,n,k", [(1, 8, 8), (1, 1024, 1024), (5, 1160, 72), (16, 128, 640), (17, 384, 1536), (33, 4096, 200), (64, 136, 4096), (64, 3072, 1024)])
def test_linear_of_few_rows(m, n, k):
    """Edges of the row, column and K tiles, every cluster size, bias, activation, pre-activation copy and residual; the sums of a
    cluster meet in a fixed order."""
    x, w, b, r = _rand((m, k), 1), _rand((n, k), 2, k ** -0.5), _rand((n,), 3), _rand((m, n), 4)
    ext = OF.load_ext()
    z = x.double() @ w.double().t() + b.double()
    near = lambda got, want: float((got.double() - want).norm() / want.norm()) < 2.0 ** -8       # one rounding of an fp32 sum
    for act, fn in ((OF.ACT_NONE, lambda t: t), (OF.ACT_GELU, torch.nn.functional.gelu), (OF.ACT_SILU, torch.nn.functional.silu)):
        y, pre = ext.linear_fwd(x, w, b, act, act != OF.ACT_NONE)
        assert near(y, fn(z)) and (act == OF.ACT_NONE or near(pre, z))
        assert torch.equal(ext.linear_fwd(x, w, b, act, False)[0], y)
    assert near(ext.linear_bias_residual(x, w, b, r), z + r.double())
    assert near(ext.linear_fwd(x, w, None, OF.ACT_NONE, False)[0], z - b.double())


@pytest.mark.parametrize("ranks", [1, 2, 4, 8])
@pytest.mark.parametrize("nt", [16, 32, 64, 128])
@pytest.mark.parametrize("n,k", [(300, 200), (136, 1032), (1032, 520)])
def test_linear_of_few_rows_every_tile_and_cluster(nt, ranks, n, k):
    """Every instantiation, whatever the rule picks: two row tiles with the last one ragged, column tiles that end inside a warp's
    four columns per lane, clusters some of whose CTAs have no k-block; the same bits in a second run."""
    m = nt + nt // 2 + 1
    x, w, b, r = _rand((m, k), 1), _rand((n, k), 2, k ** -0.5), _rand((n,), 3), _rand((m, n), 4)
    lib = ctypes.CDLL(so_path())
    ptr = lambda t: ctypes.c_void_p(0 if t is None else t.data_ptr())

    def call(act, pre, residual):
        y = torch.full((m, n), float("nan"), device="cuda", dtype=BF16)
        rc = lib.lb_gemm_small(ptr(x), ptr(w), ptr(y), m, n, k, k, k, n, ptr(b), act, ptr(pre), ptr(residual), nt, ranks,
                               ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        assert rc == 0
        return y

    z = x.double() @ w.double().t() + b.double()
    near = lambda got, want: float((got.double() - want).norm() / want.norm()) < 2.0 ** -8       # one rounding of an fp32 sum
    pre = torch.empty(m, n, device="cuda", dtype=BF16)
    y = call(OF.ACT_GELU, pre, None)
    assert near(pre, z) and near(y, torch.nn.functional.gelu(z)) and torch.equal(y, call(OF.ACT_GELU, pre, None))
    assert near(call(OF.ACT_NONE, None, r), z + r.double())


@pytest.mark.parametrize("dtype", [torch.float32, BF16])
@pytest.mark.parametrize("lens,heads,kv,d,v", [([1], 1, 1, 4, 8), ([2, 1, 17], 4, 2, 64, 64), ([16, 33], 2, 1, 128, 72), ([5, 31, 48, 7], 32, 16, 100, 128),
                                               ([40], 3, 3, 12, 136), ([9, 20], 2, 2, 60, 24)])
def test_delta_scan_two_tokens_at_a_time(lens, heads, kv, d, v, dtype):
    """Odd and even numbers of tokens, rows and columns that do not fill a block, shared key heads, states that go on; every output and
    the final state against the recurrence in 64 bits."""
    from libai_b200.inference.ragged import RaggedBatch
    from libai_b200.ops import seq_functional as SF

    tokens, kd = sum(lens), kv * d
    past = [3 * (i % 2) for i in range(len(lens))]
    rb = RaggedBatch(lens, list(range(len(lens))), past, "cuda")
    qkv, a, b = _rand((tokens, 2 * kd + heads * v), 1, 1.0, dtype), _rand((tokens, heads), 2, 1.0, dtype), _rand((tokens, heads), 3, 1.0, dtype)
    rate, bias = _rand((heads,), 4, 0.5, dtype), _rand((heads,), 5, 0.5, dtype)
    state = _rand((len(lens), heads, d, v), 6, 1.0, torch.float32)
    S = state.clone()
    out = SF.delta_scan(qkv, kd, 2 * kd, a, b, rate, bias, S, rb, kv, False)
    x, unit = qkv.double(), lambda t: t / torch.sqrt(t.square().sum(-1, keepdim=True) + 1e-6)
    q = unit(x[:, :kd].view(tokens, kv, d)).repeat_interleave(heads // kv, 1) / math.sqrt(d)
    k = unit(x[:, kd:2 * kd].view(tokens, kv, d)).repeat_interleave(heads // kv, 1)
    val, beta = x[:, 2 * kd:].view(tokens, heads, v), torch.sigmoid(b.double())
    g = torch.exp(-torch.exp(rate.double()) * torch.nn.functional.softplus(a.double() + bias.double(), threshold=200.0))
    at = 0
    for i, n in enumerate(lens):
        s = state[i].double() if past[i] else torch.zeros_like(state[i]).double()
        for t in range(at, at + n):
            s = s * g[t, :, None, None]
            u = beta[t, :, None] * (val[t] - torch.einsum("hdv,hd->hv", s, k[t]))
            s = s + k[t, :, :, None] * u[:, None]
            want = torch.einsum("hdv,hd->hv", s, q[t]).reshape(-1)
            # fp32 sums of d products per token, the state's own error carried along
            assert float((out[t].double() - want).norm()) < 2e-6 * float(want.norm()) + 2e-6 * float(s.norm()) / math.sqrt(d)
        assert float((S[i].double() - s).norm() / s.norm()) < 2e-6
        at += n


def _delta64(qkv, a, b, rate, bias, S, lens, heads, kv, d, v):
    """The recurrence token by token in float64: read-outs, final states."""
    out, final, at = [], [], 0
    for i, n in enumerate(lens):
        rows, st = qkv[at:at + n].double(), S[i].double().clone()
        q, k, val = rows[:, :kv * d].view(n, kv, d), rows[:, kv * d:2 * kv * d].view(n, kv, d), rows[:, 2 * kv * d:].view(n, heads, v)
        unit = lambda t: (t / torch.sqrt(t.square().sum(-1, keepdim=True) + 1e-6)).repeat_interleave(heads // kv, 1)
        q, k = unit(q) / math.sqrt(d), unit(k)
        beta = torch.sigmoid(b[at:at + n].double())
        g = torch.exp(-torch.exp(rate.double()) * torch.nn.functional.softplus(a[at:at + n].double() + bias.double(), threshold=300.0))
        for t in range(n):
            st = st * g[t][:, None, None]
            st = st + k[t][:, :, None] * (beta[t][:, None] * (val[t] - torch.einsum("hdv,hd->hv", st, k[t])))[:, None, :]
            out.append(torch.einsum("hdv,hd->hv", st, q[t]).reshape(-1))
        final.append(st)
        at += n
    return torch.stack(out), torch.stack(final)


@pytest.mark.parametrize("shift", [-8.0, 0.0, 6.0])
@pytest.mark.parametrize("lens,heads,kv,d,v", [([64], 1, 1, 8, 8), ([65, 3, 97], 2, 1, 64, 64), ([96, 33, 128], 6, 3, 104, 136), ([200, 64], 4, 2, 128, 72),
                                               ([70], 2, 1, 12, 16), ([95, 63, 64], 16, 8, 128, 128)])
def test_delta_scan_in_chunks(lens, heads, kv, d, v, shift):
    """Sequences on both sides of the line between chunks and pairs in one batch, last chunks of every kind, columns and rows short of
    the tiles, states carried over in slots of another order; decays near one, ordinary and near zero."""
    from libai_b200.inference.ragged import RaggedBatch
    from libai_b200.ops import seq_functional as SF

    n = sum(lens)
    qkv, a, b = _rand((n, 2 * kv * d + heads * v), 1), (_rand((n, heads), 2).float() + shift).to(BF16), _rand((n, heads), 3)
    rate, bias = _rand((heads,), 4, 0.5), _rand((heads,), 5, 0.5)
    slots, past = list(range(len(lens)))[::-1], [7 * (i % 2) for i in range(len(lens))]
    S = _rand((len(lens), heads, d, v), 6, 1.0, torch.float32)
    start = torch.stack([S[s] * (p > 0) for s, p in zip(slots, past)])
    want, final = _delta64(qkv, a, b, rate, bias, start, lens, heads, kv, d, v)
    rb = RaggedBatch(lens, slots, past, "cuda")
    run = lambda st: SF.delta_scan(qkv, kv * d, 2 * kv * d, a, b, rate, bias, st, rb, kv, False)
    first = S.clone()
    out = run(first)
    # all numbers are fp32 sums: 2^-24 per step of a product of `d` and of a chain whose links contract (decays near one keep every link's)
    assert float((out.double() - want).norm() / want.norm()) < 2.0 ** -24 * (32 + (max(lens) if shift < 0 else 0))
    assert float((first[slots].double() - final).norm() / final.norm()) < 2.0 ** -24 * (32 + (max(lens) if shift < 0 else 0))
    second = S.clone()
    assert torch.equal(run(second), out) and torch.equal(first, second)
    for i, m in enumerate(lens):                              # a sequence alone gives the same bits
        lo = sum(lens[:i])
        st, alone = S.clone(), RaggedBatch([m], [slots[i]], [past[i]], "cuda")
        rows = slice(lo, lo + m)
        y = SF.delta_scan(qkv[rows], kv * d, 2 * kv * d, a[rows], b[rows], rate, bias, st, alone, kv, False)
        assert torch.equal(y, out[rows]) and torch.equal(st[slots[i]], first[slots[i]])


@pytest.mark.parametrize("taps", [2, 3, 4])
@pytest.mark.parametrize("lens", [[173], [1, 2, 3, 4, 5, 1, 1, 160], [4, 4, 8, 130, 6, 7]])
def test_short_convolution_in_strips(lens, taps):
    """Many tokens: sequences that begin anywhere in a strip, shorter than the taps, with and without a past; the new tails."""
    from libai_b200.inference.ragged import RaggedBatch
    from libai_b200.ops import seq_functional as SF

    C, n, past = 8200, sum(lens), [5 * (i % 2) for i in range(len(lens))]
    x, w, tail = _rand((n, C + 8), 1)[:, :C], _rand((C, taps), 2), _rand((len(lens), taps - 1, C), 3)
    slots = list(range(len(lens)))[::-1]
    new, out = tail.clone(), torch.empty(n, C, device="cuda", dtype=BF16)
    SF.short_conv(x, w, new, RaggedBatch(lens, slots, past, "cuda"), out)
    at = 0
    for m, slot, p in zip(lens, slots, past):
        rows = torch.cat([tail[slot].double() * (p > 0), x[at:at + m].double()])
        z = sum(rows[j:j + m] * w[:, j].double() for j in range(taps))
        size = sum((rows[j:j + m] * w[:, j].double()).abs() for j in range(taps))
        want = z * torch.sigmoid(z)
        # fp32 sums of `taps` products, a slope of at most 1.1, one rounding to bf16
        assert bool(((out[at:at + m].double() - want).abs() <= 2.0 ** -8 * want.abs() + 2.0 ** -21 * size).all())
        assert torch.equal(new[slot].double(), rows[m:])
        at += m


@pytest.mark.parametrize("dtype", [torch.float32, BF16])
@pytest.mark.parametrize("tokens,heads,v,pad", [(1, 1, 4, 0), (37, 3, 72, 0), (200, 16, 128, 4), (5, 2, 132, 0), (3, 2, 500, 4), (9, 2, 512, 0), (9, 2, 516, 0), (9, 3, 64, 1)])
@pytest.mark.parametrize("act", [0, 1])
def test_gated_norm_of_read_outs(tokens, heads, v, pad, act, dtype):
    """Widths around the vectors of a warp, rows on and off their alignment, both gates."""
    from libai_b200.ops import seq_functional as SF

    n = heads * v
    o, gate, w, y = _rand((tokens, n), 1, 2.0, torch.float32), _rand((tokens, n + pad), 2, 1.0, dtype)[:, :n], _rand((v,), 3, 1.0, dtype), torch.empty(tokens, n + pad, device="cuda", dtype=dtype)[:, :n]
    SF.gated_rmsnorm(o, gate, w, 1e-6, act, y, heads, v)
    x, g = o.double().view(tokens, heads, v), gate.double().view(tokens, heads, v)
    want = x * torch.rsqrt(x.square().mean(-1, keepdim=True) + 1e-6) * w.double() * torch.sigmoid(g) * (g if act == 0 else 1.0)
    got = y.double().view(tokens, heads, v)
    # a dozen fp32 roundings and a sum of v squares, then one rounding to the type
    assert bool(((got - want).abs() <= (2.0 ** -20 + (2.0 ** -8 if dtype == BF16 else 0.0)) * want.abs() + 1e-30).all())


@pytest.mark.parametrize("dtype", [torch.float32, BF16])
@pytest.mark.parametrize("rows,heads,v", [(13, 5, 60), (3, 1, 64), (7, 3, 68), (1, 1, 128), (3, 3, 256), (1, 3, 260)])
def test_gated_norm_of_several_rows_per_warp(rows, heads, v, dtype):
    """Widths around 8, 16 and 32 lanes per row, last warps with rows that are not there."""
    from libai_b200.ops import seq_functional as SF

    n = heads * v
    o, gate, w, y = _rand((rows, n), 1, 2.0, torch.float32), _rand((rows, n), 2, 1.0, dtype), _rand((v,), 3, 1.0, dtype), torch.full((rows + 1, n), 3.0, device="cuda", dtype=dtype)
    SF.gated_rmsnorm(o, gate, w, 1e-6, 0, y[:rows], heads, v)
    x, g = o.double().view(rows, heads, v), gate.double().view(rows, heads, v)
    want = (x * torch.rsqrt(x.square().mean(-1, keepdim=True) + 1e-6) * w.double() * torch.sigmoid(g) * g).view(rows, n)
    # a dozen fp32 roundings and a sum of v squares, then one rounding to the type
    assert bool(((y[:rows].double() - want).abs() <= (2.0 ** -20 + (2.0 ** -8 if dtype == BF16 else 0.0)) * want.abs() + 1e-30).all())
    assert bool((y[rows] == 3).all())


@pytest.mark.parametrize("value", [float("inf"), float("nan"), 3e38])
def test_delta_scan_in_chunks_value_that_is_not_finite(value):
    """It reaches no earlier token, no other column and no other head."""
    from libai_b200.inference.ragged import RaggedBatch
    from libai_b200.ops import seq_functional as SF

    heads, kv, d, v, n, at = 2, 1, 64, 72, 100, 75
    qkv, a, b = _rand((n, 2 * kv * d + heads * v), 1), _rand((n, heads), 2), _rand((n, heads), 3)
    rate, bias, rb = _rand((heads,), 4, 0.5), _rand((heads,), 5, 0.5), RaggedBatch([n], [0], [0], "cuda")

    def run(x):
        S = torch.zeros(1, heads, d, v, device="cuda")
        return SF.delta_scan(x, kv * d, 2 * kv * d, a, b, rate, bias, S, rb, kv, False).view(n, heads, v), S[0]

    out, S = run(qkv)
    x = qkv.clone()
    x[at, 2 * kv * d + v + 5] = value                         # head 1, column 5
    got, T = run(x)
    other = torch.ones(heads, v, dtype=torch.bool, device="cuda")
    other[1, 5] = False
    assert torch.equal(got[:, other], out[:, other]) and torch.equal(T.transpose(1, 2)[other], S.transpose(1, 2)[other])
    # earlier tokens of the chunk take these sums in another order
    near = (got[:at, 1, 5] - out[:at, 1, 5]).abs().max()
    assert float(near) < 2.0 ** -20 * float(out[:at, 1].abs().max()) and torch.equal(got[:64, 1, 5], out[:64, 1, 5])
    assert not torch.isfinite(got[at:, 1, 5]).all() if value != 3e38 else torch.isfinite(got[at, 1, 5])


def _delta_case(lens, heads, kv, d, v, shift):
    n = sum(lens)
    return (_rand((n, 2 * kv * d + heads * v), 1), (_rand((n, heads), 2).float() + shift).to(BF16), _rand((n, heads), 3), _rand((heads,), 4, 0.5),
            _rand((heads,), 5, 0.5))


@pytest.mark.parametrize("shift", [-8.0, -3.0, 0.0, 5.0])
@pytest.mark.parametrize("lens,heads,kv,d,v", [([257, 130], 4, 2, 128, 128), ([88, 96, 97, 640], 2, 2, 64, 64)])
def test_delta_scan_in_chunks_is_as_exact_as_token_by_token(lens, heads, kv, d, v, shift):
    """The same numbers in rows off the vectors' alignment are scanned token by token in fp32: chunks are no further from 64 bits."""
    from libai_b200.inference.ragged import RaggedBatch
    from libai_b200.ops import seq_functional as SF

    qkv, a, b, rate, bias = _delta_case(lens, heads, kv, d, v, shift)
    start = _rand((len(lens), heads, d, v), 6, 1.0, torch.float32)
    want, final = _delta64(qkv, a, b, rate, bias, start, lens, heads, kv, d, v)
    rb = RaggedBatch(lens, list(range(len(lens))), [1] * len(lens), "cuda")
    wide = torch.zeros(qkv.shape[0], qkv.shape[1] + 3, device="cuda", dtype=BF16)
    wide[:, :-3] = qkv
    errors = []
    for rows in (qkv, wide[:, :-3]):
        S = start.clone()
        out = SF.delta_scan(rows, kv * d, 2 * kv * d, a, b, rate, bias, S, rb, kv, False)
        errors.append((float((out.double() - want).norm() / want.norm()), float((S.double() - final).norm() / final.norm())))
    assert errors[0][0] <= errors[1][0] and errors[0][1] <= errors[1][1], errors


@pytest.mark.parametrize("value", [float("nan"), float("inf")])
@pytest.mark.parametrize("where", ["a", "b", "key", "query"])
def test_delta_scan_in_chunks_input_that_is_not_finite(where, value):
    """A gate, key or query that is not finite reaches no earlier token and no head that does not read it."""
    from libai_b200.inference.ragged import RaggedBatch
    from libai_b200.ops import seq_functional as SF

    heads, kv, d, v, lens, at = 4, 2, 64, 72, [100, 90], 75
    qkv, a, b, rate, bias = _delta_case(lens, heads, kv, d, v, 0.0)
    rb = RaggedBatch(lens, [0, 1], [0, 0], "cuda")

    def run(qkv, a, b):
        S = torch.zeros(2, heads, d, v, device="cuda")
        return SF.delta_scan(qkv, kv * d, 2 * kv * d, a, b, rate, bias, S, rb, kv, False).view(-1, heads, v), S

    out, S = run(qkv, a, b)
    x, ga, gb = qkv.clone(), a.clone(), b.clone()
    hit = [2, 3]                                              # the second key head's
    if where == "a":
        ga[at, 2], hit = value, [2]
    elif where == "b":
        gb[at, 2], hit = -value, [2]
    else:
        x[at, (d if where == "query" else kv * d + d) + 5] = value
    got, T = run(x, ga, gb)
    rest = [h for h in range(heads) if h not in hit]
    assert torch.equal(got[:, rest], out[:, rest]) and torch.equal(T[:, rest], S[:, rest])           # other heads
    assert torch.equal(got[100:], out[100:]) and torch.equal(T[1], S[1])                             # the other sequence
    assert torch.equal(got[:64], out[:64])                                                           # earlier chunks
    # earlier tokens of the chunk may take their sums in another order
    assert float((got[64:at, hit] - out[64:at, hit]).abs().max()) < 2.0 ** -20 * float(out[64:at].abs().max())


def test_delta_scan_in_chunks_vectors_beyond_fp32_squares():
    """A key or query whose squares overflow counts as zero, as in the scan token by token."""
    from libai_b200.inference.ragged import RaggedBatch
    from libai_b200.ops import seq_functional as SF

    heads, kv, d, v, n = 2, 1, 128, 64, 110
    qkv, a, b, rate, bias = _delta_case([n], heads, kv, d, v, 0.0)
    rb, results = RaggedBatch([n], [0], [1], "cuda"), []
    for size in (0.0, 2e38):
        x = qkv.clone()
        x[40, d:2 * d] = size                                 # key
        x[70, :d] = -size                                     # query
        S = _rand((1, heads, d, v), 6, 1.0, torch.float32)
        results.append((SF.delta_scan(x, kv * d, 2 * kv * d, a, b, rate, bias, S, rb, kv, False), S))
    assert torch.equal(results[0][0], results[1][0]) and torch.equal(results[0][1], results[1][1])


@pytest.mark.parametrize("dtype", [torch.float32, BF16])
@pytest.mark.parametrize("n", [1, 17])
def test_delta_scan_value_that_is_not_finite(n, dtype):
    """An infinite value in the last of an odd number of tokens: its own column of the state becomes infinite with the sign of the key
    (no pair partner that is not there may turn it into a NaN), the other columns stay what they are without it."""
    from libai_b200.inference.ragged import RaggedBatch
    from libai_b200.ops import seq_functional as SF

    kv, heads, d, v = 1, 2, 64, 64
    qkv, a, b = _rand((n, 2 * d + heads * v), 1, 1.0, dtype), _rand((n, heads), 2, 1.0, dtype), _rand((n, heads), 3, 1.0, dtype)
    rate, bias = _rand((heads,), 4, 0.5, dtype), _rand((heads,), 5, 0.5, dtype)
    rb = RaggedBatch([n], [0], [0], "cuda")

    def run(x):
        S = torch.zeros(1, heads, d, v, device="cuda")
        return SF.delta_scan(x, d, 2 * d, a, b, rate, bias, S, rb, kv, False), S[0]

    base = run(qkv)
    x = qkv.clone()
    x[-1, 2 * d + v + 5] = float("inf")                       # head 1, column 5
    out, S = run(x)
    key = x[-1, d:2 * d].float()
    assert torch.equal(S[1, :, 5], torch.where(key > 0, 1.0, -1.0) * float("inf"))
    assert not torch.isfinite(out[-1, v + 5]) and not torch.isnan(out[-1, v + 5])
    keep = torch.ones(heads, v, dtype=torch.bool, device="cuda")
    keep[1, 5] = False
    assert torch.equal(S.transpose(1, 2)[keep], base[1].transpose(1, 2)[keep])
    assert torch.equal(out[-1].view(heads, v)[keep], base[0][-1].view(heads, v)[keep]) and torch.equal(out[:-1], base[0][:-1])


@pytest.mark.parametrize("lens", [False, True])
@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("b,s,a", [(1, 1, 1), (2, 63, 2), (1, 64, 3), (2, 65, 1), (1, 127, 2), (3, 128, 1), (1, 130, 2), (2, 333, 4), (1, 1024, 16)])
def test_attention_backward_head_dim_128(b, s, a, causal, lens):
    """Lengths around the 64-query and 128-key tiles, causal, full and right-padded."""
    qkv, go = _rand((b, s, a, 384), 1).requires_grad_(True), _rand((b, s, a, 128), 2)
    n = torch.tensor([max(1, s - 37 * i) for i in range(b)], dtype=torch.int32, device="cuda") if lens else None
    y = OF.attention_qkvpacked(qkv, causal=causal, scale=0.09, kv_lens=n)
    y.backward(go)
    x = qkv.detach().double().requires_grad_(True)
    keep = torch.ones(b, 1, s, s, dtype=torch.bool, device="cuda")
    keep = keep.tril() if causal else keep
    if lens:
        keep = keep & (torch.arange(s, device="cuda")[None, None, None] < n[:, None, None, None])
    # a causal query always sees key 0, which every sequence has
    _attend64(*(t.permute(0, 2, 1, 3) for t in x.split(128, -1)), 0.09, keep).permute(0, 2, 1, 3).backward(go.double())
    for got, want in zip(qkv.grad.split(128, -1), x.grad.split(128, -1)):
        # probabilities and their gradients pass through bf16, then the result does; where everything cancels (one key) the bf16 result's own scale
        assert float((got.double() - want).norm()) < 2.0 ** -7 * float(want.norm()) + 2.0 ** -9 * float(go.norm()) * (s == 1)


@pytest.mark.parametrize("causal", [False, True])
def test_attention_backward_head_dim_128_repeats(causal):
    """dK and dV are sums in a fixed order inside one CTA: the same bits every time (a tile must not be taken with the row statistics
    of an earlier one: 18 query tiles go through three stages and two groups of warps)."""
    qkv, go = _rand((4, 1100, 16, 384), 1).requires_grad_(True), _rand((4, 1100, 16, 128), 2)
    y = OF.attention_qkvpacked(qkv, causal=causal, scale=128 ** -0.5)
    first = torch.autograd.grad(y, qkv, go, retain_graph=True)[0][..., 128:]
    for _ in range(4):
        assert torch.equal(torch.autograd.grad(y, qkv, go, retain_graph=True)[0][..., 128:], first)


@pytest.mark.parametrize("M", [40, 129, 1100, 2500])
@pytest.mark.parametrize("layout", [0, 1])
@pytest.mark.parametrize("wide", [False, True])
def test_gemm_tile_order_in_bands(M, layout, wide):
    """B of 25 MB (row by row) and beyond 48 MB: bands of row blocks, a last band of one block, ragged edges.  Whole numbers below 256:
    exact in bf16."""
    N, K = (49176 if wide else 24600, 520) if layout == 0 else (264, 98312 if wide else 49160)
    g = torch.Generator(device="cuda").manual_seed(M)
    x = torch.randint(-1, 2, (M, K), generator=g, device="cuda").to(BF16)
    w = torch.randint(-1, 2, (N, K) if layout == 0 else (K, N), generator=g, device="cuda").to(BF16)
    if layout == 1:
        x[:, 512:-8] = 0        # sums stay below 256
    want = x.float() @ (w.float().t() if layout == 0 else w.float())
    assert want.abs().max() < 256
    assert torch.equal(OF.load_ext().gemm(x, w, layout, None, None, False, BF16).float(), want)


_W = lambda *s, i=1: _rand(s, i, s[-1] ** -0.5)
_ROT = lambda s, d: (torch.linspace(0, 3, s * d, device="cuda").view(s, d).cos().contiguous(), torch.linspace(0, 3, s * d, device="cuda").view(s, d).sin().contiguous())
_GRAPHLESS = {
    "linear": lambda x: OF.linear(x, _W(72, 64), _rand((72,), 2), "gelu"),
    "mlp": lambda x: OF.mlp(x, _W(128, 64), _rand((128,), 2), _W(64, 128, i=3), "gelu", _rand((64,), 4), x),
    "mlp_without_residual": lambda x: OF.mlp(x, _W(128, 64), _rand((128,), 2), _W(64, 128, i=3)),
    "linear_bias_residual": lambda x: OF.linear_bias_residual(x, _W(64, 64), _rand((64,), 2), x),
    "layer_norm": lambda x: OF.layer_norm(x, _rand((64,), 2), _rand((64,), 3)),
    "layer_norm_with_skip": lambda x: OF.layer_norm_with_skip(x, _rand((64,), 2), _rand((64,), 3)),
    "rms_norm": lambda x: OF.rms_norm(x, _rand((64,), 2)),
    "bias_act": lambda x: OF.bias_act(x, _rand((64,), 2)),
    "bias_add": lambda x: OF.bias_dropout_add(x, _rand((64,), 2), _rand((3, 40, 64), 3), 0.0, False),
    "gated_mlp": lambda x: gated_mlp(x, *_W(256, 64).split(128), _W(64, 128, i=3)),
    "swiglu": lambda x: OF.swiglu(x, _rand((3, 40, 64), 2)),
    "attention_64": lambda x: OF.attention(*(_rand((3, 4, 40, 64), i) + x.mean() for i in range(3)), causal=True),
    "attention_48": lambda x: OF.attention(*(_rand((3, 4, 40, 48), i) + x.mean() for i in range(3)), causal=True),
    "attention_packed": lambda x: OF.attention_packed("qkv", (_rand((3, 40, 4, 96), 1) + x.mean(),), causal=False, scale=0.2),
    "attention_qkvpacked": lambda x: OF.attention_qkvpacked(_rand((3, 40, 4, 192), 1) + x.mean(), causal=True, scale=0.2),
    "rotary": lambda x: OF.apply_rotary(x.view(3, 40, 1, 64).permute(0, 2, 1, 3).contiguous(), *_ROT(40, 64)),
    "rotary_qkv": lambda x: OF.apply_rotary_qkv(_rand((3, 40, 4, 96), 1) + x.mean(), *_ROT(64, 32)),
    "cross_entropy": lambda x: OF.vocab_parallel_cross_entropy(x.clone(), torch.arange(120, device="cuda").view(3, 40) % 64),
    "embedding": lambda x: OF.embedding(torch.arange(30, device="cuda") % 40, x[0]),
}


@pytest.mark.parametrize("name", sorted(_GRAPHLESS))
def test_calls_without_a_graph_equal_those_with_one(name):
    """Without gradients the forwards run past the autograd functions: the same bits, nothing kept, nothing that asks for a gradient."""
    x = _rand((3, 40, 64), 9)
    one = lambda y: y[0] if isinstance(y, tuple) else y
    with_graph = one(_GRAPHLESS[name](x.clone().requires_grad_(True)))
    assert with_graph.requires_grad
    for mode in (torch.no_grad, torch.inference_mode):
        with mode():
            got = one(_GRAPHLESS[name](x.clone().requires_grad_(True)))
            assert not got.requires_grad and got.grad_fn is None and got.shape == with_graph.shape and torch.equal(got, with_graph.detach())


@pytest.mark.parametrize("grad", [False, True])
@pytest.mark.parametrize("d", [24, 48])
def test_attention_transformed_differentiated_forward_and_traced(d, grad):
    """vmap, both forward modes, tracing and tensors without memory see the unfused operators, in gradient mode and out of it."""
    scale = d ** -0.5
    q, k, v, t = (_rand((2, 3, 20, d), i) for i in range(4))
    f = lambda x: OF.attention(x, k, v, causal=True, scale=scale)
    ref = lambda x: OF.attention_ref(x, k, v, causal=True, scale=scale)
    near = lambda a, b: float((a.double() - b.double()).norm() / b.double().norm()) < 2.0 ** -7
    with torch.set_grad_enabled(grad):
        assert near(torch.func.vmap(f)(torch.stack([q, t])), torch.stack([ref(q), ref(t)]))
        packed = lambda x: OF.attention_packed("qkv", (x,), causal=False, scale=scale) is None
        told = []
        torch.func.vmap(lambda x: (told.append(packed(x)), x)[1])(_rand((2, 1, 20, 3, 3 * d), 5))
        assert told == [True]
        want = torch.func.jvp(ref, (q,), (t,))
        assert all(near(a, b) for a, b in zip(torch.func.jvp(f, (q,), (t,)), want))
        with torch.autograd.forward_ad.dual_level():
            out = torch.autograd.forward_ad.unpack_dual(f(torch.autograd.forward_ad.make_dual(q, t)))
            assert near(out.primal, want[0]) and near(out.tangent, want[1])
        traced = torch.jit.trace(f, (q,), check_trace=False)
        assert near(traced(t), ref(t))
        with FakeTensorMode():
            x = torch.empty(2, 3, 20, d, dtype=BF16, device="cuda")
            assert OF.attention(x, x, x, causal=True).shape == x.shape
            assert OF.attention_cached(x[:, :, :1], x[:, :, :1], x[:, :, :1], x, x, scale=scale) is None


@pytest.mark.parametrize("d", [48, 64, 128])
@pytest.mark.parametrize("pin", [False, True])
def test_attention_backward_from_tensors_saved_on_the_host(d, pin):
    """Saved-tensor hooks may give tensors back with other strides."""
    q, k, v = (_rand((2, 3, 40, d), i).requires_grad_(True) for i in range(3))
    go = _rand((2, 3, 40, d), 4)
    want = torch.autograd.grad(OF.attention(q, k, v, causal=True), (q, k, v), go)
    with torch.autograd.graph.save_on_cpu(pin_memory=pin):
        out = OF.attention(q, k, v, causal=True)
    assert all(torch.equal(a, b) for a, b in zip(torch.autograd.grad(out, (q, k, v), go), want))


def _gpt_block(heads, dim, mask="causal", **kw):
    from libai_b200.layers import TransformerLayer
    from libai_b200.layers._param import param_defaults
    from libai_b200.layers.attention import AttnMaskType

    with param_defaults(dtype=BF16, device="cuda", seed=3):
        m = TransformerLayer(heads * dim, 3 * heads * dim, heads, attn_mask_type=getattr(AttnMaskType, mask), **kw)
    with torch.no_grad():
        for i, p in enumerate(m.parameters()):
            p.copy_(_rand(p.shape, i, 0.05) + (1.0 if i in (0, 6) else 0.0))
    return m.eval()


def _llama_block(heads, dim, joint):
    from libai_b200.layers._param import param_defaults
    from libai_b200.models.llama_model import LlamaDecoderLayer

    with param_defaults(dtype=BF16, device="cuda", seed=3):
        m = LlamaDecoderLayer(heads * dim, 2 * heads * dim, heads, qkv_bias=joint)
    with torch.no_grad():
        for i, p in enumerate(m.parameters()):
            p.copy_(_rand(p.shape, i, 0.05) + (1.0 if p.dim() == 1 and p.shape[0] == heads * dim else 0.0))
        if joint:                                              # side by side, as an optimizer's flat buffer has them
            g, u = m.mlp.gate_proj, m.mlp.up_proj
            both = torch.cat([g.weight, u.weight])
            g.weight.data, u.weight.data = both[:g.weight.shape[0]], both[g.weight.shape[0]:]
    return m.eval()


def _by_modules(m, call):
    """The same call with a hook that has to see a module (one without a residual of its own): the modules run one by one."""
    seen = []
    handle = (m.mlp if hasattr(m, "self_attention") else m.post_attention_layernorm).register_forward_hook(lambda *a: seen.append(1))
    out = call()
    handle.remove()
    assert seen
    return out


def _flat(out):
    return [out] if torch.is_tensor(out) else [out[0], *out[1]]


@pytest.mark.parametrize("past", [None, 1, 70])
@pytest.mark.parametrize("b,s,heads,dim,mask", [(1, 1, 4, 24, "causal"), (2, 37, 16, 24, "causal"), (3, 130, 3, 64, "causal"), (1, 200, 2, 128, "padding"),
                                                (2, 65, 4, 48, "padding"), (1, 9, 1, 72, "causal")])
def test_block_without_a_graph_in_one_call(b, s, heads, dim, mask, past):
    """The native call and the modules: the same bits, with and without a cache; head dims that neither attention takes as well."""
    m = _gpt_block(heads, dim, mask)
    x = _rand((b, 1 if past else s, heads * dim), 1)
    kv = None if past is None else tuple(_rand((b, heads, past, dim), 5 + i) for i in range(2))
    with torch.no_grad():
        for use_cache in (False, True):
            call = lambda: m(x, past_key_value=kv, use_cache=use_cache)
            for got, want in zip(_flat(call()), _flat(_by_modules(m, call))):
                assert torch.equal(got, want) and got.stride() == want.stride() and not got.requires_grad
        y = m(x.transpose(0, 1).contiguous().transpose(0, 1), past_key_value=kv)
        assert torch.equal(y, m(x, past_key_value=kv))


@pytest.mark.parametrize("joint", [False, True])
@pytest.mark.parametrize("past", [None, 1, 70])
@pytest.mark.parametrize("b,s,heads,dim", [(1, 1, 4, 64), (2, 70, 3, 128), (3, 33, 2, 48)])
def test_llama_block_without_a_graph_in_one_call(b, s, heads, dim, past, joint):
    m = _llama_block(heads, dim, joint)
    x = _rand((b, 1 if past else s, heads * dim), 1)
    kv = None if past is None else tuple(_rand((b, heads, past, dim), 5 + i) for i in range(2))
    cos, sin = _ROT(128, dim)
    with torch.no_grad():
        for use_cache in (False, True):
            call = lambda: m(x, past_key_value=kv, cos_cached=cos, sin_cached=sin, use_cache=use_cache)
            for got, want in zip(_flat(call()), _flat(_by_modules(m, call))):
                assert torch.equal(got, want) and got.stride() == want.stride() and not got.requires_grad


@pytest.mark.parametrize("joint", [False, True])
@pytest.mark.parametrize("b,s,heads,dim", [(1, 40, 4, 64), (2, 130, 2, 128)])
def test_llama_block_residuals_in_the_epilogues(b, s, heads, dim, joint):
    """Residual adds in the projections' epilogues and skip gradients in the norms' backward against additions of their own (hooks on
    attention and MLP keep those)."""
    m, (cos, sin) = _llama_block(heads, dim, joint), _ROT(256, dim)
    x, gy = _rand((b, s, heads * dim), 1), _rand((b, s, heads * dim), 2)

    def run():
        xi = x.clone().requires_grad_(True)
        y = m(xi, cos_cached=cos, sin_cached=sin)
        return [y, *torch.autograd.grad(y, [xi, *m.parameters()], gy)]

    got = run()
    hooks = [k.register_forward_hook(lambda *a: None) for k in (m.self_attn, m.mlp, m.input_layernorm, m.post_attention_layernorm)]
    for u, v in zip(got, run()):
        # bf16 roundings of the sums (2^-8 each) that are not taken any more, through one block
        assert u.shape == v.shape and float((u.detach().double() - v.detach().double()).norm()) < 2.0 ** -6 * float(v.detach().double().norm())
    for h in hooks:
        h.remove()


def test_block_in_one_call_leaves_everything_else_to_the_modules():
    """Masks, active dropout, replaced forwards, replaced modules, functional parameters, transforms, graph capture."""
    from libai_b200.layers import MLP

    m, x = _gpt_block(4, 64), _rand((2, 40, 256), 1)
    with torch.no_grad():
        base = m(x)
        keep = torch.ones(2, 1, 40, 40, dtype=torch.bool, device="cuda").tril()
        assert float((m(x, keep) - base).float().norm()) < 2.0 ** -7 * float(base.float().norm())
        d = _gpt_block(4, 64, output_dropout_prob=0.5)
        assert torch.equal(d(x), base) and not torch.equal(d.train()(x), base)
        old, calls = MLP.forward, []
        try:
            MLP.forward = lambda self, *a, **k: (calls.append(1), old(self, *a, **k))[1]
            assert torch.equal(m(x), base) and calls
        finally:
            MLP.forward = old
        m.mlp.forward = lambda h, residual=None: residual
        assert not torch.equal(m(x), base)
        del m.mlp.forward
        half = {k: (v * 0.5 if v.dim() == 2 else v).detach() for k, v in m.named_parameters()}
        assert not torch.equal(torch.func.functional_call(m, half, (x,)), base)
        assert torch.equal(torch.func.vmap(lambda t: t * 2)(x), x * 2) and torch.equal(m(x), base)
        side = torch.cuda.Stream()
        with torch.cuda.stream(side):
            m(x)
        side.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            y = m(x)
        graph.replay()
        assert torch.equal(y, base)
    assert m(x).requires_grad


@pytest.mark.parametrize("scale", [1.0, 0.25])
@pytest.mark.parametrize("size,poison", [(1e-3, None), (3.0, None), (3.0, float("nan")), (3.0, float("inf")), (0.0, None)])
def test_gradient_norm_and_clip_coefficient_over_groups(size, poison, scale):
    """One accumulator for all parameter groups, coefficient below and at one, what is not finite, a loss scale."""
    from libai_b200.optim import AdamW, get_default_optimizer_params

    m = torch.nn.Sequential(torch.nn.Linear(72, 40), torch.nn.LayerNorm(40), torch.nn.Linear(40, 8)).cuda().to(BF16)
    opt = AdamW(get_default_optimizer_params(m, weight_decay_norm=0.0, weight_decay_bias=0.0, clip_grad_max_norm=1.0, clip_grad_norm_type=2.0), lr=1e-3)
    opt.setup()
    assert sum(g is not None for g in opt._groups) > 1
    for i, p in enumerate(m.parameters()):
        p.main_grad.copy_(_rand(p.shape, i, size, torch.float32))
    if poison is not None:
        next(m.parameters()).main_grad[3, 5] = poison
    opt.grad_scale = scale
    want = torch.sqrt(sum(p.main_grad.double().square().sum() for p in m.parameters())) * scale
    norm = opt.clip_grad()
    assert norm.dim() == 0 and norm.dtype == torch.float32 and opt._clip_coef.dim() == 0
    coef = torch.clamp(1.0 / (want + 1e-6), max=1.0)
    # sums of a few thousand squares in fp32 and a handful of roundings
    assert torch.allclose(norm.double(), want, rtol=1e-5, equal_nan=True) and torch.allclose(opt._clip_coef.double(), coef, rtol=1e-5, equal_nan=True)


@pytest.mark.parametrize("where", ["stream", "side stream", "capture"])
@pytest.mark.parametrize("make,b,s", [(lambda: _gpt_block(16, 24, "causal"), 1, 40), (lambda: _gpt_block(4, 64, "causal"), 3, 260),
                                      (lambda: _gpt_block(6, 48, "padding"), 2, 150), (lambda: _llama_block(4, 64, True), 2, 130)])
def test_launches_that_start_before_the_last_one_ends(make, b, s, where):
    """Ten passes in a row, each on the last one's output and in memory that the one before left, and one backward pass: the same bits as with a wait after
    every operator (the operators' sums have one order; only weight gradients do not)."""
    m = make()
    h = next(m.parameters()).numel()
    x = _rand((b, s, h), 1)
    kw = {}
    if type(m).__name__ == "LlamaDecoderLayer":
        kw = dict(zip(("cos_cached", "sin_cached"), _ROT(512, 64)))

    class Waiting(torch.utils._python_dispatch.TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            out = func(*args, **(kwargs or {}))
            torch.cuda.synchronize()
            return out

    def forward():
        y = x
        for _ in range(10):
            y = m(y, **kw)
        return y

    def backward():
        xi = x.clone().requires_grad_(True)
        return torch.autograd.grad(m(xi, **kw), xi, x)[0]

    with torch.no_grad(), Waiting():
        want = forward()
    stream = torch.cuda.current_stream() if where == "stream" else torch.cuda.Stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.no_grad(), torch.cuda.stream(stream):
        for _ in range(3):
            got = forward()
        if where == "capture":
            stream.synchronize()
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph, stream=stream):
                got = forward()
            for _ in range(3):
                got.zero_()
                graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(got, want)
    if x.shape[-1] == 6 * 48:                       # (attention that adds dQ up in one order)
        with Waiting():
            want = backward()
        with torch.cuda.stream(stream):
            got = backward()
        torch.cuda.synchronize()
        assert torch.equal(got, want)


@pytest.mark.parametrize("vocab", [8, 2056, 8184, 8192, 8200, 18440, 50304, 1003])
def test_cross_entropy_statistics_in_groups_of_loads(vocab):
    """Maxima are exact.  A thread adds up ``vocab / 256`` terms in two sums, 13 more come from the other threads: as many roundings of 2^-24 at most, and each
    exponential is off by 2 ulp and the rounding of its argument, up to 2^-24 of 60.  A row may be minus infinity almost everywhere."""
    x = _rand((5, vocab), 1, 4.0)
    x[1] -= 40.0
    x[2, : vocab // 2] = float("-inf")
    x[2, vocab // 3] = 1.0
    x[3, vocab - 1] = 50.0
    labels = torch.tensor([0, vocab - 1, vocab, -1, vocab // 2], device="cuda")
    mx, se, tgt = load_ext().ce_stats(x, labels, 0)
    d = x.double()
    want = (d - d.amax(1, keepdim=True)).exp().sum(1)
    assert torch.equal(mx, x.float().amax(1))
    assert torch.equal(tgt, torch.stack([x[0, 0], x[1, -1], x.new_zeros(()), x.new_zeros(()), x[4, vocab // 2]]).float())
    assert float(((se.double() - want).abs() / want).max()) <= (vocab / 256 + 13 + 4 + 60) * 2.0 ** -24
    x[4, vocab // 3] = float("nan")
    assert bool(load_ext().ce_stats(x, labels, 0)[1][4].isnan())


@pytest.mark.parametrize("m,n,k", [(2049, 16, 2048), (2560, 128, 2048), (8192, 64, 4096), (8193, 64, 4096), (4096, 8, 4096), (4097, 24, 4104), (2560, 136, 2048)])
def test_many_rows_against_one_tile_of_columns(m, n, k):
    """Both sides of the rule that gives such products to clusters along K: bf16 results within the rounding of the result (2^-8 of it) and of ``k`` fp32
    additions (``k * 2^-24`` of the sum of magnitudes; the tensor core truncates, twice that)."""
    x, w, b = _rand((m, k), 1), _rand((n, k), 2), _rand((n,), 3)
    y = load_ext().linear_fwd(x, w, b, 0, False)[0]
    want = x.double() @ w.double().T + b.double()
    bound = want.abs() * 2.0 ** -8 + (x.double().abs() @ w.double().abs().T + b.double().abs()) * k * 2.0 ** -23
    assert bool(((y.double() - want).abs() <= bound).all())
    assert float((y.double() - want).norm() / want.norm()) < 2.0 ** -8


@pytest.mark.parametrize("dim,b,s,a,biased,causal", [(64, 3, 100, 4, False, False), (64, 5, 128, 2, False, True), (128, 2, 384, 4, False, False), (64, 2, 304, 3, True, False),
                                                     (128, 2, 264, 2, True, True), (64, 4, 520, 2, False, False)])
def test_attention_lengths_written_by_the_launch_before(dim, b, s, a, biased, causal):
    """Key lengths, and the memory they are in, change right before the kernel that reads them: the same bits as with a wait in between, forward and
    backward (without a bias), one and two tiles per block."""
    qkv = _rand((b, s, a, 3 * dim), 1)
    q, k, v = (t.permute(0, 2, 1, 3) for t in qkv.split(dim, -1))
    bias = _rand((b, a, s, s), 2) if biased else None
    go, base, n = _rand((b, s, a, dim), 3), torch.arange(b, device="cuda", dtype=torch.int32) * 17, torch.empty(b, device="cuda", dtype=torch.int32)

    def run(wait):
        out = []
        for i in range(6):
            torch.add(base, 1 + s * i // 6, out=n)
            if wait:
                torch.cuda.synchronize()
            if biased:
                o, lse, _ = load_ext().attn_fwd(q, k, v, causal, dim ** -0.5, n, bias, None, 0.0, 0)
                out += [o, lse]
            else:
                x = qkv.detach().requires_grad_(True)
                o = OF.attention_qkvpacked(x, causal=causal, scale=dim ** -0.5, kv_lens=n)
                out += [o.detach(), *(torch.autograd.grad(o, x, go)[0].split(dim, -1)[1:])]           # dK and dV have a fixed order
            if wait:
                torch.cuda.synchronize()
        return out

    want = run(True)
    for _ in range(3):
        assert all(torch.equal(x, y) for x, y in zip(run(False), want))
    assert not torch.equal(want[0], want[-2 if biased else -3])


def _waiting():
    """Mode that waits for the device after every operator."""
    class Waiting(torch.utils._python_dispatch.TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            out = func(*args, **(kwargs or {}))
            torch.cuda.synchronize()
            return out

    return Waiting()


def _chain_fp8():
    out, w = [], _rand((264, 512), 9)
    for i, (m, size) in enumerate([(300, 1.0), (300, 40.0), (64, 0.01), (300, 7.0), (2000, 300.0)]):
        xq, dx = load_ext().quantize_e4m3(_rand((m, 512), i, size))
        wq, dw = load_ext().quantize_e4m3(w * (i + 1))
        out.append(load_ext().linear_fp8_fwd(xq, wq, dx, dw, None, 0, False, None)[0])
    return out


def _chain_loss():
    from libai_b200.layers import LMLogits, ParallelCrossEntropyLoss

    out, w = [], _rand((4104, 256), 1, 0.05).requires_grad_(True)
    for i, m in enumerate([700, 33, 700, 1500]):
        x = _rand((1, m, 256), 2 + i).requires_grad_(True)
        labels = torch.randint(0, 4104, (1, m), device="cuda", generator=torch.Generator("cuda").manual_seed(i))
        loss = ParallelCrossEntropyLoss()(LMLogits(4104)(x, w), labels)
        out += [loss.detach(), torch.autograd.grad(loss.sum(), x)[0]]
    return out


def _chain_attention(drop):
    out = []
    for i, (s, d) in enumerate([(136, 64), (264, 128), (520, 64), (136, 64)]):
        torch.manual_seed(i)
        q, k, v = (t + 0.25 for t in _rand((2, 4, 3 * s, d), i).split(s, 2))
        bias = None if drop else _rand((1, 4, s, s), 7 + i) * 2.0
        out.append(OF.attention(q, k, v, causal=True, bias=bias, dropout_p=0.2 * drop, training=bool(drop)))
    return out


def _chain_block(dim):
    m, x, out = _gpt_block(4, dim), _rand((3, 200, 4 * dim), 1).requires_grad_(True), []
    y = x
    for _ in range(4):
        y = m(y)
        out.append(y.detach())
    y.sum().backward()                              # the kernels in a row; its sums over blocks have no fixed order
    return out


@pytest.mark.parametrize("chain", [_chain_fp8, _chain_loss, lambda: _chain_attention(0), lambda: _chain_attention(1), lambda: _chain_block(64),
                                   lambda: _chain_block(128)], ids=["fp8", "loss", "bias", "dropout", "block 64", "block 128"])
def test_inputs_written_by_the_launch_before(chain):
    """Scales, logits, scores' bias and activations straight from the kernel before, in memory that was something else a moment ago: the same bits as
    with a wait after every operator."""
    with _waiting():
        want = chain()
    for _ in range(3):
        got = chain()
        assert len(got) == len(want) and all(torch.equal(a, b) for a, b in zip(got, want))


@pytest.mark.parametrize("rows", [3, 200, 2100])
def test_residual_that_begins_anywhere(rows):
    """A block's input may be a view off the vectors of 16 bytes that the epilogue loads: few rows and many, fp8, and a whole block forward and backward."""
    h, k = 192, 256
    x, w, b, flat = _rand((rows, k), 1), _rand((h, k), 2, 0.1), _rand((h,), 3), _rand((rows * h + 8,), 4)
    xq, dx = load_ext().quantize_e4m3(x)
    wq, dw = load_ext().quantize_e4m3(w)
    for off in (1, 2, 4):
        view = flat[off:off + rows * h].view(rows, h)
        assert view.data_ptr() % 16
        assert torch.equal(load_ext().linear_bias_residual(x, w, b, view), load_ext().linear_bias_residual(x, w, b, view.clone()))
        assert torch.equal(load_ext().linear_fp8_fwd(xq, wq, dx, dw, b, 0, False, view)[0], load_ext().linear_fp8_fwd(xq, wq, dx, dw, b, 0, False, view.clone())[0])
    if rows == 200:
        m, (cos, sin) = _llama_block(3, 64, False), _ROT(256, 64)
        results = []
        for x in (flat[3:3 + rows * h].view(1, rows, h), flat[3:3 + rows * h].view(1, rows, h).clone()):
            x = x.detach().requires_grad_(True)
            y = m(x, cos_cached=cos, sin_cached=sin)
            results.append((y.detach().double(), torch.autograd.grad(y, x, y.detach())[0].double()))
        for got, want in zip(*results):              # another norm kernel reads rows off their alignment: roundings of its result (2^-8) through the block
            assert float((got - want).norm()) < 2.0 ** -6 * float(want.norm())


@pytest.mark.parametrize("m,n,k", [(8, 8, 64), (24, 264, 72), (128, 256, 512), (200, 72, 2664), (384, 1160, 2048), (1152, 384, 4096), (4104, 1024, 520)])
def test_weight_gradient_accumulates_in_boxes(m, n, k):
    """dW += dyᵀ x through boxes of 32 x 32 with rows and columns behind the end, split along K and not, into a slice of a larger buffer
    whose other elements stay as they are."""
    a, b = _rand((k, m), 1), _rand((k, n), 2)
    buf = _rand((m + 2, n + 8), 3, dtype=torch.float32)
    before = buf.clone()
    load_ext().gemm(a, b, 2, None, buf[1:m + 1, 4:n + 4], True, torch.float32)
    old = before[1:m + 1, 4:n + 4].double()
    want = old + a.double().t() @ b.double()
    # k products and k / 16 additions, none of which is more than one unit of 24 bits of the sum of magnitudes off
    bound = (k / 16 + 2) * 2.0 ** -23 * (old.abs() + a.double().abs().t() @ b.double().abs())
    assert bool(((buf[1:m + 1, 4:n + 4].double() - want).abs() <= bound).all())
    buf[1:m + 1, 4:n + 4] = before[1:m + 1, 4:n + 4]
    assert torch.equal(buf, before)


@pytest.mark.parametrize("bn", [64, 128, 192, -128, -192, -256])
@pytest.mark.parametrize("layout", [0, 1, 2])
@pytest.mark.parametrize("m,n,k", [(129, 136, 64), (256, 192, 72), (300, 200, 840), (1400, 1160, 136), (2500, 776, 264)])
def test_gemm_tiles_of_every_width(bn, layout, m, n, k):
    """Single CTAs' tiles and CTA pairs' (negative), whatever the rule picks: rows and columns that end inside a tile and inside a pair's half, one wave and
    several, nothing written behind the last column.  Whole numbers, exact in every format."""
    if layout == 2:
        m = (m + 7) // 8 * 8
    if layout == 2 and bn in (64, 128, 192) and n < bn // 2:
        pytest.skip("not a tile for so few columns")
    g = torch.Generator(device="cuda").manual_seed(m + n)
    ints = lambda *s: (torch.rand(*s, generator=g, device="cuda") < 0.2).to(BF16) * torch.randint(-1, 2, s, generator=g, device="cuda").to(BF16)
    a, b = ints(*((k, m) if layout == 2 else (m, k))), ints(*((n, k) if layout == 0 else (k, n)))
    out = torch.full((m, n + 8), 3.0, device="cuda", dtype=torch.float32 if layout == 2 else BF16)
    lib = ctypes.CDLL(so_path())
    ptr = lambda t: ctypes.c_void_p(t.data_ptr())
    rc = lib.lb_gemm_bf16(ptr(a), ptr(b), ptr(out), m, n, k, a.shape[1], b.shape[1], n + 8, layout, 2 if layout == 2 else 0, ctypes.c_void_p(0), 0,
                          ctypes.c_void_p(0), bn, 0, ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == 0
    want = (a.float().t() if layout == 2 else a.float()) @ (b.float().t() if layout == 0 else b.float())
    assert want.abs().max() < 256
    assert torch.equal(out[:, :n].float(), want + (3.0 if layout == 2 else 0.0)) and bool((out[:, n:] == 3).all())


@pytest.mark.parametrize("m,k,ns", [(1, 64, [8]), (129, 128, [16, 8]), (300, 72, [136, 16, 264]), (2500, 264, [384, 384, 192, 24]), (2500, 520, [512, 512, 256, 16, 8]),
                                    (1000, 128, [8, 256, 264, 120, 192, 200, 16, 1032]), (600, 4104, [6144, 16])])
def test_products_with_several_matrices_in_one_launch(m, k, ns):
    """Every width of tile, up to eight matrices that end inside a tile, several waves, bands of rows; nothing written behind the last column.  Whole numbers, exact in
    every format."""
    g = torch.Generator(device="cuda").manual_seed(m + k)
    ints = lambda *s: (torch.rand(*s, generator=g, device="cuda") < 0.2).to(BF16) * torch.randint(-1, 2, s, generator=g, device="cuda").to(BF16)
    a, ws = ints(m, k + 8)[:, 8:], [ints(n, k) for n in ns]
    total = sum(ns)
    out = torch.full((m, total + 8), 3.0, device="cuda", dtype=BF16)
    lib = ctypes.CDLL(so_path())
    ptrs, cols = (ctypes.c_void_p * len(ns))(*[w.data_ptr() for w in ws]), (ctypes.c_int * len(ns))(*ns)
    rc = lib.lb_gemm_multi(ctypes.c_void_p(a.data_ptr()), ptrs, cols, len(ns), ctypes.c_void_p(out.data_ptr()), m, k, k + 8, total + 8,
                           ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == 0
    want = a.float() @ torch.cat(ws).float().t()
    assert want.abs().max() < 256
    assert torch.equal(out[:, :total].float(), want) and bool((out[:, total:] == 3).all())


def _train_block(kind, dim, with_main_grad, s=40):
    """A block, its call and its inputs: causal, right-padded, without a mask, T5 decoder, Llama; causal with a mask of its own, which stands in the triangle's place (dense,
    padded on the left) or, in the flash kernels, beside it (right-padded)."""
    from libai_b200.layers import TransformerLayer
    from libai_b200.layers._param import param_defaults
    from libai_b200.layers.attention import AttnMaskType, KeyPaddingMask
    from libai_b200.models.llama_model import LlamaDecoderLayer, rotary_tables
    from libai_b200.optim import AdamW, get_default_optimizer_params

    heads = 4
    hidden = heads * dim
    with param_defaults(dtype=BF16, device="cuda", seed=1):
        if kind == "llama":
            layer = LlamaDecoderLayer(hidden, 256, heads, rms_norm_eps=1e-6, max_position_embeddings=max(64, s))
        else:
            layer = TransformerLayer(hidden, 2 * hidden, heads, is_decoder=kind == "decoder",
                                     attn_mask_type=AttnMaskType.causal if kind.startswith("causal") else AttnMaskType.padding)
        for i, p in enumerate(layer.parameters()):
            p.data.copy_(_rand(p.shape, 10 + i, 0.05 if p.dim() > 1 else 0.1) + (p.dim() == 1))
    if with_main_grad or kind == "llama":       # (one buffer: gate and up weights side by side)
        opt = AdamW(get_default_optimizer_params(layer), lr=1e-3)
        opt.setup()
    x = _rand((3, s, hidden), 2).requires_grad_(True)
    if kind == "llama":
        cos, sin = rotary_tables(dim, max(64, s), device="cuda")
        return layer, lambda: layer(x, cos_cached=cos, sin_cached=sin), [x]
    if kind == "decoder":
        enc = _rand((3, 24, hidden), 3).requires_grad_(True)
        m = torch.ones(3, 1, s, s, dtype=torch.bool, device="cuda").tril()
        cm = (torch.arange(24, device="cuda") < 20).expand(3, 1, s, 24)
        return layer, lambda: layer(x, m, enc, cm), [x, enc]
    mask = KeyPaddingMask((torch.arange(s, device="cuda")[None] < torch.tensor([[s], [17], [1]], device="cuda")).long()) if kind.endswith("padded") else None
    if kind == "causal-left":
        mask = KeyPaddingMask((torch.arange(s, device="cuda")[None] >= torch.tensor([[0], [17], [s - 1]], device="cuda")).long())
    if kind == "causal-prefix":                 # the first 13 positions see one another
        mask = torch.ones(s, s, dtype=torch.bool, device="cuda").tril()
        mask[:13, :13] = True
    return layer, lambda: layer(x, mask), [x]


@pytest.mark.parametrize("main_grad", [False, True])
@pytest.mark.parametrize("kind,dim", [("causal", 64), ("causal", 24), ("padded", 128), ("padded", 48), ("none", 32), ("decoder", 32), ("decoder", 64), ("llama", 128),
                                      ("causal-prefix", 48), ("causal-prefix", 64), ("causal-padded", 24), ("causal-padded", 64), ("causal-left", 32), ("causal-left", 64)])
def test_block_graph_in_one_call(kind, dim, main_grad):
    """One node per block, one per operator (a hook on a module) and the Python functions (a dispatch mode looks on) launch the same kernels: outputs to
    the bit, gradients up to the order of their sums; a second backward pass, checkpointing and frozen parameters work as with the modules, and create_graph gives the same gradients
    (constants: the test below)."""
    from torch.utils._python_dispatch import TorchDispatchMode
    from torch.utils.checkpoint import checkpoint

    class Look(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            return func(*args, **(kwargs or {}))

    def grads(how):
        layer, call, inputs = _train_block(kind, dim, main_grad)
        params = list(layer.parameters())
        if how == "nodes":
            layer.input_layernorm.register_forward_hook(lambda *a: None)
        if how == "python":
            with Look():
                y = call()
        elif how == "checkpoint":
            y = checkpoint(lambda *_: call(), *inputs, use_reentrant=False)
        else:
            y = call()
        assert ("Block" in type(y.grad_fn).__name__ or "Block" in y.grad_fn.name()) == (how in ("block", "checkpoint")), y.grad_fn.name()
        gy = _rand(y.shape, 5)
        y.backward(gy, retain_graph=True)
        if how == "block":
            y.backward(gy)                       # twice: all gradients double
        out = [t.grad for t in inputs] + [p.main_grad if getattr(p, "main_grad", None) is not None else p.grad for p in params]
        assert all(g is not None for g in out) and all(p.grad_added_to_main_grad for p in params if getattr(p, "main_grad", None) is not None)
        return y.detach(), [g.double() / (2 if how == "block" else 1) for g in out]

    want, wg = grads("python")
    for how in ("block", "nodes", "checkpoint"):
        y, got = grads(how)
        assert torch.equal(y, want)
        for a, b in zip(got, wg):
            # one bf16 rounding of an operator's result (2^-9) where sums met in another order, a few operators deep
            assert float((a - b).norm()) <= 2.0 ** -7 * float(b.norm()), how
    layer, call, inputs = _train_block(kind, dim, main_grad)
    for p in layer.mlp.parameters():
        p.requires_grad_(False)
    y = call()
    assert "Block" not in y.grad_fn.name()
    y.backward(_rand(y.shape, 5))
    assert float((inputs[0].grad.double() - wg[0]).norm()) <= 2.0 ** -7 * float(wg[0].norm())
    layer, call, inputs = _train_block(kind, dim, main_grad)
    y = call()
    g = torch.autograd.grad(y, inputs, _rand(y.shape, 5), create_graph=True)
    assert float((g[0].double() - wg[0]).norm()) <= 2.0 ** -7 * float(wg[0].norm())


@pytest.mark.parametrize("kind,dim", [("causal-prefix", 48), ("causal-prefix", 64), ("causal-padded", 24), ("causal-padded", 128), ("causal-left", 64), ("padded", 48)])
def test_block_trains_the_function_that_it_evaluates(kind, dim):
    """With a mask: as one node, with a node per operator (frozen parameters) and without a graph, to the bit."""
    layer, call, _ = _train_block(kind, dim, False)
    with torch.no_grad():
        want = call()
    y = call()
    assert "Block" in y.grad_fn.name() and torch.equal(y, want)
    layer.mlp.dense_4h_to_h.bias.requires_grad_(False)
    y = call()
    assert "Block" not in y.grad_fn.name() and torch.equal(y, want)


@pytest.mark.parametrize("main_grad", [False, True])
@pytest.mark.parametrize("kind,dim", [("causal", 64), ("padded", 48), ("decoder", 32), ("llama", 128)])
def test_block_under_hooks_that_copy_what_is_saved(kind, dim, main_grad):
    """Saved tensors that come back as copies (offloading): gradients as without the hooks."""
    got = []
    for hooks in (False, True):
        layer, call, inputs = _train_block(kind, dim, main_grad)
        if hooks:
            with torch.autograd.graph.save_on_cpu():
                y = call()
        else:
            y = call()
        assert "Block" in y.grad_fn.name()
        y.backward(_rand(y.shape, 5))
        got.append([t.grad for t in inputs] + [p.main_grad if getattr(p, "main_grad", None) is not None else p.grad for p in layer.parameters()])
    for a, b in zip(*got):
        assert float((a.double() - b.double()).norm()) <= 2.0 ** -7 * float(a.double().norm())


@pytest.mark.parametrize("kind,dim", [("causal", 64), ("llama", 128)])
def test_block_graph_takes_biases_that_changed_in_between(kind, dim):
    """They are no part of the backward pass."""
    layer, call, inputs = _train_block(kind, dim, True)
    y = call()
    with torch.no_grad():
        for m in layer.modules():
            if getattr(m, "bias", None) is not None:
                m.bias.add_(1)
    y.backward(_rand(y.shape, 5))
    assert inputs[0].grad is not None


@pytest.mark.parametrize("kind,dim", [("causal", 64), ("causal-prefix", 48), ("decoder", 32), ("llama", 128)])
def test_block_gradients_with_create_graph_are_constants(kind, dim):
    """As one node, with a node per operator and from the Python functions: the gradients of an ordinary pass, without a graph of their own."""
    from torch.utils._python_dispatch import TorchDispatchMode

    class Look(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            return func(*args, **(kwargs or {}))

    for how in ("block", "nodes", "python"):
        layer, call, inputs = _train_block(kind, dim, False)
        if how == "nodes":
            layer.input_layernorm.register_forward_hook(lambda *a: None)
        if how == "python":
            with Look():
                y = call()
        else:
            y = call()
        params = [p for p in layer.parameters() if getattr(p, "main_grad", None) is None]
        gy = _rand(y.shape, 5)
        got = torch.autograd.grad(y, inputs + params, gy, create_graph=True)
        want = torch.autograd.grad(y, inputs + params, gy)
        for a, b in zip(got, want):
            assert not a.requires_grad and float((a.double() - b.double()).norm()) <= 2.0 ** -7 * float(b.double().norm()), how


@pytest.mark.parametrize("recompute", [False, True])
@pytest.mark.parametrize("kind,dim", [("causal", 64), ("causal-prefix", 48), ("decoder", 48), ("llama", 128)])
def test_block_graph_holds_no_more_than_its_operators(kind, dim, recompute):
    """Peak of memory of a pass forward and one back, as one node and with a node per operator: what is saved goes when its operator is done (and with checkpointing hooks when it is made)."""
    from torch.utils.checkpoint import checkpoint

    peak = []
    for how in ("nodes", "block"):
        layer, call, inputs = _train_block(kind, dim, True, 512)
        if how == "nodes":
            layer.input_layernorm.register_forward_hook(lambda *a: None)
        step = (lambda: checkpoint(lambda *_: call(), *inputs, use_reentrant=False)) if recompute else call
        step().sum().backward()
        for t in inputs:
            t.grad = None
        gc.collect()                             # (what earlier tests left must not go in between)
        torch.cuda.synchronize()
        stat = lambda which: torch.cuda.memory_stats()["requested_bytes.all." + which]       # (allocated ones count the whole of a cached block)
        base, peak_of = stat("current"), []
        torch.cuda.reset_peak_memory_stats()
        y = step()
        peak_of.append(stat("peak") - base)
        gy = _rand(y.shape, 5)
        torch.cuda.reset_peak_memory_stats()
        y.backward(gy)
        peak_of.append(stat("peak") - base)
        peak.append(peak_of)
        assert ("Block" in y.grad_fn.name()) == (how == "block")
        del y, gy
    unit = inputs[0].numel() * 2                  # a [tokens, width] tensor in bf16; statistics and the like apart
    assert all(b <= n + unit / 4 for n, b in zip(*peak)), [[round(v / unit, 2) for v in p] for p in peak]


def test_block_graph_refuses_what_changed_in_between():
    layer, call, inputs = _train_block("causal", 64, True)
    y = call()
    with torch.no_grad():
        layer.mlp.dense_4h_to_h.weight.add_(1)
    with pytest.raises(RuntimeError, match="modified by an inplace operation"):
        y.backward(_rand(y.shape, 5))
    y = call()
    y.backward(_rand(y.shape, 5))
    with pytest.raises(RuntimeError, match="second time"):
        y.backward(_rand(y.shape, 5))


@pytest.mark.parametrize("kind", ["causal", "none", "padded", "stripes"])
@pytest.mark.parametrize("b,sq,sk,a,d", [(5, 300, 300, 16, 24), (30, 130, 260, 8, 48), (2, 128, 128, 150, 32), (37, 256, 256, 4, 64)])
def test_split_attention_of_many_work_items(b, sq, sk, a, d, kind):
    """Several work items per CTA, rows of the mask that are visible, masked or mixed for 32 or 64 keys at a time: as close to 64 bits as the unfused form, the same
    bits again."""
    if kind == "causal" and sk < sq:
        pytest.skip("more queries than keys under a causal mask: unfused form")
    m = None
    if kind == "padded":
        nq, nk = (torch.randint(1, n + 1, (b,), device="cuda", generator=torch.Generator(device="cuda").manual_seed(n)) for n in (sq, sk))
        m = ((torch.arange(sq, device="cuda") < nq[:, None])[:, None, :, None] & (torch.arange(sk, device="cuda") < nk[:, None])[:, None, None, :])
    if kind == "stripes":
        m = ((torch.arange(sq, device="cuda") // 32)[:, None] + torch.arange(sk, device="cuda") // 64) % 3 != 0
        m[sq // 3, sk // 2] ^= True
    causal = kind == "causal" and d != 64         # (head dim 64 takes these kernels with a mask only)
    if d == 64 and m is None:
        m = torch.ones(sq, sk, dtype=torch.bool, device="cuda")
        m = m.tril(sk - sq) if kind == "causal" else m
    q, k, v, go = _rand((b, a, sq, d), 1), _rand((b, sk, a, d), 2).permute(0, 2, 1, 3), _rand((b, a, sk, d), 3), _rand((b, a, sq, d), 4)
    keep = torch.ones(sq, sk, dtype=torch.bool, device="cuda").tril(sk - sq) if causal else m
    x = [t.double().requires_grad_(True) for t in (q, k, v)]
    s = x[0] @ x[1].transpose(-1, -2) * 0.3
    if keep is not None:
        s = s.masked_fill(~keep, float("-inf") if causal else -10000.0)
    want = torch.softmax(s, -1) @ x[2]
    want.backward(go.double())
    far = []
    for fn in (OF.attention, OF.attention_ref):
        t = [y.detach().clone().requires_grad_(True) for y in (q, k, v)]
        y = fn(*t, causal=causal, scale=0.3, mask=m)
        y.backward(go)
        far.append([float((u.double() - w).norm() / w.norm()) for u, w in zip((y, *(z.grad for z in t)), (want, *(z.grad for z in x)))])
        if fn is OF.attention:
            first = [z.grad for z in t]
            again = torch.autograd.grad(OF.attention(*t, causal=causal, scale=0.3, mask=m), t, go)
            assert all(torch.equal(u, w) for u, w in zip(first, again))
    # the bf16 result's rounding is most of both; the sums of 32-bit products meet in another order
    assert all(got < 1.05 * ref + 1e-5 for got, ref in zip(*far)), far


@pytest.mark.parametrize("rms", [False, True])
@pytest.mark.parametrize("m", [1, 2, 3, 4, 5, 8, 9, 16])
@pytest.mark.parametrize("n,k", [(40, 8), (136, 1032), (1152, 384), (3072, 1024), (6144, 2048), (520, 4096)])
def test_linear_of_few_rows_behind_a_norm(n, k, m, rms):
    """Statistics by 8 to 128 threads per row, rows and k-blocks that end early, clusters with empty CTAs; rows with a large common part, which a sum of squares would not survive."""
    x, g, b = _rand((m, k), 1) * 2 + 50, 1 + 0.1 * _rand((k,), 2), None if rms else _rand((k,), 3)
    w, bias = _rand((n, k), 4, k ** -0.5), _rand((n,), 5)
    y = torch.full((m + 1, n), 7.0, device="cuda", dtype=BF16)
    ptr = lambda t: ctypes.c_void_p(0 if t is None else t.data_ptr())
    rc = ctypes.CDLL(so_path()).lb_gemm_small_norm(ptr(x), ptr(g), ptr(b), ctypes.c_float(1e-5), int(rms), ptr(w), ptr(y), m, n, k, k, k, n, ptr(bias), 0,
                                                   ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == 0
    d = x.double()
    d = d * torch.rsqrt(d.square().mean(-1, keepdim=True) + 1e-5) * g.double() if rms else torch.nn.functional.layer_norm(d, (k,), g.double(), b.double(), 1e-5)
    want = d.to(BF16).double() @ w.double().t() + bias.double()
    # the normalised rows are rounded to bf16 once (some a step off, where 32 and 64 bits round apart), the result once
    assert float((y[:m].double() - want).norm()) < 2.0 ** -8 * float(want.norm()) and bool((y[m] == 7).all())


@pytest.mark.parametrize("which", ["both", "before", "behind"])
@pytest.mark.parametrize("rows", [1, 5, 131, 600, 1900])
@pytest.mark.parametrize("h", [8, 264, 768, 1000, 1024])
def test_norm_backward_with_the_biases_around_it(h, rows, which):
    """Every width of vectors per lane, rows of a warp from none to several, results added to what the buffers hold; result and column sums against float64."""
    gy, x, gadd, gamma = _rand((rows, h), 1), _rand((rows, h), 2) + 3, _rand((rows, h), 3), 1 + 0.1 * _rand((h,), 4)
    ext = load_ext()
    _, mean, rstd = ext.norm_fwd(x, gamma, torch.zeros_like(gamma), 1e-5, False)
    sums = [_rand((h,), 5 + i, dtype=torch.float32) for i in range(4)]
    old = [t.double() for t in sums]
    gx = torch.full((rows + 1, h), 7.0, device="cuda", dtype=BF16)
    ptr = lambda t: ctypes.c_void_p(0 if t is None else t.data_ptr())
    rc = ctypes.CDLL(so_path()).lb_norm_bwd_sums(ptr(gy), ptr(x), ptr(gamma), ptr(mean), ptr(rstd), ptr(gx), ptr(sums[0]), ptr(sums[1]), rows, h, ptr(gadd),
                                                 ptr(sums[2] if which != "before" else None), ptr(sums[3] if which != "behind" else None),
                                                 ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == 0
    x64 = x.double().requires_grad_(True)
    g64, b64 = gamma.double().requires_grad_(True), torch.zeros(h, device="cuda", dtype=torch.float64, requires_grad=True)
    torch.nn.functional.layer_norm(x64, (h,), g64, b64, 1e-5).backward(gy.double())
    want = x64.grad + gadd.double()
    assert float((gx[:rows].double() - want).norm()) < 2.0 ** -8 * float(want.norm()) + 1e-6 and bool((gx[rows] == 7).all())
    for got, was, d, n in ((sums[0], old[0], g64.grad, gy.double().abs().sum(0) * 4), (sums[1], old[1], b64.grad, gy.double().abs().sum(0)),
                           (sums[2], old[2], gadd.double().sum(0) * (which != "before"), gadd.double().abs().sum(0)),
                           (sums[3], old[3], gx[:rows].double().sum(0) * (which != "behind"), gx[:rows].double().abs().sum(0))):
        # fp32 sums: a rounding of 2^-24 of the magnitudes per term of a chain of at most rows / 4, and of the normalised x (2^-20)
        assert bool(((got.double() - was - d).abs() <= (2.0 ** -20 + rows * 2.0 ** -26) * (n + was.abs() + 1)).all())


@pytest.mark.parametrize("batch", [4, 40])
@pytest.mark.parametrize("kind", ["gpt", "llama"])
def test_launches_of_a_generation_step_are_counted(kind, batch):
    """One kernel or two for a norm and the product behind it: the count is what the device ran."""
    from libai_b200 import ops
    from libai_b200.layers import TransformerLayer
    from libai_b200.layers._param import param_defaults
    from libai_b200.layers.attention import AttnMaskType
    from libai_b200.models.llama_model import LlamaDecoderLayer, rotary_tables

    with param_defaults(dtype=BF16, device="cuda", seed=1):
        layer = (TransformerLayer(512, 2048, 8, attn_mask_type=AttnMaskType.causal) if kind == "gpt"
                 else LlamaDecoderLayer(512, 1024, 8, rms_norm_eps=1e-6, max_position_embeddings=64)).eval()
    x, past = _rand((batch, 1, 512), 1), (_rand((batch, 8, 20, 64), 2), _rand((batch, 8, 20, 64), 3))
    kw = {}
    if kind == "llama":
        kw["cos_cached"], kw["sin_cached"] = rotary_tables(64, 64, device="cuda")
    with torch.no_grad():
        step = lambda: layer(x, past_key_value=past, use_cache=True, **kw)
        step()
        with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
            before = ops.launch_count()
            step()
            counted = ops.launch_count() - before
            torch.cuda.synchronize()
    ran = sum(e.count for e in prof.key_averages() if "lb::" in e.key)
    assert counted == ran > 0


@pytest.mark.parametrize("main_grad", [False, True])
@pytest.mark.parametrize("rms", [False, True])
@pytest.mark.parametrize("h", [64, 1000, 1280, 12288])
def test_norm_of_no_rows(h, rms, main_grad):
    """An empty batch forward and back: empty results, zeros for the parameters."""
    x = torch.empty(0, h, device="cuda", dtype=BF16, requires_grad=True)
    w, b = (torch.nn.Parameter(_rand((h,), i)) for i in (1, 2))
    for p in (w, b):
        if main_grad:
            p.main_grad = torch.full((h,), 3.0, device="cuda")
    y = OF.rms_norm(x, w) if rms else OF.layer_norm(x, w, b)
    y.backward(torch.empty_like(y))
    assert y.shape == x.grad.shape == (0, h)
    for p in (w,) if rms else (w, b):
        assert bool((p.main_grad == 3).all()) if main_grad else bool((p.grad == 0).all())


def test_residual_stream_off_its_alignment_refuses_nothing_for_later():
    """A stream that TMA cannot write takes the other product; the next one of those sizes, on its 16 bytes, does not."""
    from libai_b200.ops import seq_functional as SF

    a, w, buf = _rand((40, 64), 1), _rand((24, 64), 2), _rand((40 * 24 + 1,), 3, dtype=torch.float32)
    before = set(SF._GEMM_REFUSED)
    for off in (1, 0):
        x = buf[off:off + 40 * 24].view(40, 24)
        want = x.double() + a.double() @ w.double().t()
        SF.linear_accumulate(x, a, w)
        # (the product passes through bf16 where the stream is off its alignment)
        assert float((x.double() - want).norm()) < (2.0 ** -8 if off else 2.0 ** -20) * float(want.norm())
    assert SF._GEMM_REFUSED == before
