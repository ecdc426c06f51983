"""Timed cases: the single layers and calls that training and generation with this package are made of.

Every case is a dict of plain values; ``prepare`` builds what a program has in hand before the call (layers with their weights, the
optimizer that owns the parameters, inputs, masks, caches), ``run`` makes one pass through public entry points and returns all of its
outputs, ``exact`` gives the same outputs in 64 bits from plain torch.  Sizes come from the recipes under ``configs/`` and
``projects/`` and from ``bench.py``; ``draw`` spreads over the ranges that they span, odd lengths among them.

Kinds:
  block    ``TransformerLayer`` forward + backward (GPT: causal, BERT: right-padded batch, ViT: no mask), gradients in the flat buffers
  decoder  the same layer as a T5 decoder block: dense 0/1 self and cross masks, another length on the encoder side
  llama    ``LlamaDecoderLayer`` forward + backward (RMS norm, rotary, SwiGLU, head dim 128)
  attend   ``attention_qkvpacked`` forward + backward, up to long sequences
  decode   one generation step of a ``TransformerLayer`` / ``LlamaDecoderLayer`` with a key/value cache
  head     tied LM head + vocab-parallel cross entropy, forward + backward
  adamw    ``AdamW.step`` with gradient clipping on the parameters of a few blocks (bf16 parameters, fp32 master copy)
  gpt      a whole ``GPTModel`` call: token ids to logits
  delta    prompt pass of the gated delta-rule mixer over a ragged batch
"""
import math

import numpy as np
import torch

from libai_b200.config import DictConfig
from libai_b200.layers import LMLogits, ParallelCrossEntropyLoss, TransformerLayer, VocabEmbedding
from libai_b200.layers._param import param_defaults
from libai_b200.layers.attention import AttnMaskType, KeyPaddingMask
from libai_b200.layers.delta_rule import GatedDeltaMixer
from libai_b200.inference.ragged import RaggedBatch
from libai_b200.models.gpt_model import GPTModel
from libai_b200.models.llama_model import LlamaDecoderLayer, rotary_tables
from libai_b200.ops import functional as OF
from libai_b200.optim import AdamW, get_default_optimizer_params
from libai_b200.utils import distributed as dutil

DEVICE = "cuda"
BF16 = torch.bfloat16


# ------------------------------------------------------------------------------------------------------------------ cases
def listed():
    return [
        # one block of the benchmark GPT-2 (nl24 h1024 a16 s1024, micro-batch 8)
        dict(name="gpt_block", kind="block", mask="causal", batch=8, seq=1024, heads=16, dim=64, ffn=4096),
        # one block of the BERT pre-training recipe: 16 heads of 48, padded batch of 16
        dict(name="bert_block_padded", kind="block", mask="padded", batch=16, seq=512, heads=16, dim=48, ffn=4096),
        # one block of ViT-Large/16 at 224 x 224: 197 tokens
        dict(name="vit_block", kind="block", mask="none", batch=64, seq=197, heads=16, dim=64, ffn=4096),
        # one decoder block of the T5 recipe (12 heads of 32, batch 16, 512 encoder and 128 decoder tokens)
        dict(name="t5_decoder_block", kind="decoder", batch=16, seq=128, enc=512, heads=12, dim=32, ffn=1536),
        # one block of Llama-2 7B, one sequence of 2048 tokens
        dict(name="llama_block", kind="llama", batch=1, seq=2048, heads=32, dim=128, ffn=11008),
        # long-context self-attention, head dim 128
        dict(name="attention_long", kind="attend", causal=True, batch=1, seq=8192, heads=16, dim=128),
        # one generated token per sequence, GPT-2 block, 8 sequences with half of the context filled
        dict(name="gpt_decode", kind="decode", model="gpt", batch=8, past=511, heads=16, dim=64, ffn=4096),
        # one generated token per sequence, Llama-2 7B block, 4 sequences near the end of the context
        dict(name="llama_decode", kind="decode", model="llama", batch=4, past=2046, heads=32, dim=128, ffn=11008),
        # LM head and loss of the benchmark GPT-2
        dict(name="lm_head_loss", kind="head", batch=8, seq=1024, hidden=1024, vocab=50304),
        # optimizer step over four blocks of the benchmark GPT-2 (50 M parameters)
        dict(name="adamw_step", kind="adamw", layers=4, heads=16, dim=64, ffn=4096),
        # prompt through the whole GPT-2 of the pre-training recipe (nl6 h384 a16), logits of every position
        dict(name="gpt_prompt", kind="gpt", layers=6, batch=1, seq=200, heads=16, dim=24, ffn=1536, vocab=50304),
        # prompt pass of a delta-rule mixer of the serving benchmark (width 2048), ragged batch
        dict(name="delta_prompt", kind="delta", width=2048, heads=16, kv_heads=8, dim=128, sequences=4, longest=1024),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["block", "block", "block", "decoder", "llama", "attend", "decode", "decode", "head", "adamw", "gpt", "delta"])
    if kind == "block":
        dim = rng.choice([24, 32, 48, 64, 64, 128])
        heads = rng.choice([h for h in (4, 6, 8, 12, 16, 20) if 192 <= h * dim <= 1536])
        seq = rng.choice([_log(rng, 33, 1500), 8 * _log(rng, 8, 128)])
        batch = max(1, min(128, _log(rng, 128, 8192) // seq))
        return dict(kind=kind, mask=rng.choice(["causal", "padded", "none"]), batch=batch, seq=seq, heads=heads, dim=dim, ffn=4 * heads * dim)
    if kind == "decoder":
        heads, dim = rng.choice([(12, 32), (16, 48), (8, 64), (12, 64), (16, 64)])
        return dict(kind=kind, batch=rng.randint(1, 16), seq=rng.randint(17, 160), enc=rng.choice([rng.randint(33, 512), 8 * rng.randint(4, 64)]),
                    heads=heads, dim=dim, ffn=8 * rng.randint(96, 384))
    if kind == "llama":
        heads = rng.choice([8, 16, 24, 32])
        return dict(kind=kind, batch=rng.randint(1, 2), seq=_log(rng, 65, 1024), heads=heads, dim=128, ffn=128 * (heads * 8 // 3))
    if kind == "attend":
        dim, seq = rng.choice([64, 128]), _log(rng, 129, 8192)
        heads = rng.choice([8, 12, 16])
        batch = max(1, min(16, 8192 // seq))
        return dict(kind=kind, causal=rng.random() < 0.7, batch=batch if seq < 4096 else 1, seq=seq, heads=heads, dim=dim)
    if kind == "decode":
        if rng.random() < 0.5:
            heads, dim = rng.choice([(16, 24), (16, 64), (12, 64), (20, 64)])
            return dict(kind=kind, model="gpt", batch=_log(rng, 1, 64), past=_log(rng, 16, 1023), heads=heads, dim=dim, ffn=4 * heads * dim)
        heads = rng.choice([8, 16, 32])
        return dict(kind=kind, model="llama", batch=_log(rng, 1, 16), past=_log(rng, 16, 2047), heads=heads, dim=128, ffn=128 * (heads * 8 // 3))
    if kind == "head":
        hidden = rng.choice([384, 768, 1024, 1280])
        tokens = _log(rng, 200, 8192 * 1024 // hidden if hidden > 1024 else 8192)
        batch = rng.choice([1, 2, 4, 8])
        return dict(kind=kind, batch=batch, seq=max(1, tokens // batch), hidden=hidden, vocab=rng.choice([21128, 30592, 32000, 50304]))
    if kind == "adamw":
        heads = rng.choice([6, 12, 16, 20])
        return dict(kind=kind, layers=rng.randint(1, 4), heads=heads, dim=64, ffn=256 * heads)
    if kind == "gpt":
        heads, dim = rng.choice([(16, 24), (12, 32), (12, 64)])
        batch = rng.randint(1, 4)
        return dict(kind=kind, layers=rng.randint(2, 6), batch=batch, seq=_log(rng, 17, 1024), heads=heads, dim=dim, ffn=4 * heads * dim,
                    vocab=rng.choice([21128, 30592, 50304]))
    heads = rng.choice([8, 16])
    return dict(kind=kind, width=128 * heads, heads=heads, kv_heads=rng.choice([heads // 2, heads]), dim=128, sequences=rng.randint(1, 8),
                longest=_log(rng, 30, 1024))


# ----------------------------------------------------------------------------------------------------------------- inputs
class _Rng:
    """Values on the device, from the seed alone."""

    def __init__(self, seed):
        self.g = torch.Generator(device=DEVICE)
        self.g.manual_seed(int(seed) * 7919 + 13)

    def normal(self, shape, std, dtype=BF16, mean=0.0):
        return torch.empty(tuple(shape), dtype=torch.float32, device=DEVICE).normal_(mean, std, generator=self.g).to(dtype)

    def ints(self, shape, hi, lo=0):
        return torch.randint(lo, hi, tuple(shape), device=DEVICE, generator=self.g)


def _weights(rng, module):
    """Trained-like values: matrices N(0, 0.02²) like the recipes' initialisers leave them, norms around one, small biases."""
    with torch.no_grad():
        for name, p in module.named_parameters():
            if p.dim() >= 2:
                p.copy_(rng.normal(p.shape, 0.02))
            elif name.endswith("weight"):
                p.copy_(rng.normal(p.shape, 0.1, mean=1.0))
            else:
                p.copy_(rng.normal(p.shape, 0.02))


def _lengths(count, longest, seed, shortest):
    """Valid lengths of a batch, the longest among them."""
    r = np.random.RandomState((int(seed) * 31 + 7) % (2 ** 31))
    n = r.randint(min(shortest, longest), longest + 1, count)
    n[0] = longest
    return [int(v) for v in n]


def _optimizer(module):
    """The optimizer owns the parameters: weight gradients go into its flat fp32 buffers (``main_grad``)."""
    opt = AdamW(get_default_optimizer_params(module, weight_decay_norm=0.0, weight_decay_bias=0.0, clip_grad_max_norm=1.0,
                                             clip_grad_norm_type=2.0), lr=1e-4, weight_decay=0.01)
    opt.setup()
    return opt


def _layer(case):
    if case["kind"] in ("llama",) or case.get("model") == "llama":
        return LlamaDecoderLayer(case["heads"] * case["dim"], case["ffn"], case["heads"], rms_norm_eps=1e-6, max_position_embeddings=2048)
    return TransformerLayer(case["heads"] * case["dim"], case["ffn"], case["heads"], is_decoder=case["kind"] == "decoder",
                            layernorm_epsilon=1e-5, apply_query_key_layer_scaling=True,
                            attn_mask_type=AttnMaskType.causal if case.get("mask") == "causal" or case["kind"] in ("decode", "adamw")
                            else AttnMaskType.padding)


def prepare(case, seed):
    dutil.reset_dist_util()
    rng, kind, s = _Rng(seed), case["kind"], {"case": case}
    with param_defaults(dtype=BF16, device=DEVICE, seed=1):
        if kind in ("block", "decoder", "llama", "decode"):
            hidden = case["heads"] * case["dim"]
            layer = s["layer"] = _layer(case)
            _weights(rng, layer)
            n = 1 if kind == "decode" else case["seq"]
            s["x"] = rng.normal((case["batch"], n, hidden), 1.0)
            if case.get("model") == "llama" or kind == "llama":
                s["cos"], s["sin"] = rotary_tables(case["dim"], 4096, device=DEVICE)
            if kind == "decode":
                shape = (case["batch"], case["heads"], case["past"], case["dim"])
                s["past"] = (rng.normal(shape, 0.7), rng.normal(shape, 0.7))
                layer.eval()
                return s
            s["gy"] = rng.normal(s["x"].shape, 1.0)
            s["opt"] = _optimizer(layer)
            s["params"] = dict(layer.named_parameters())
            s["x"].requires_grad_(True)
            if kind == "block" and case["mask"] == "padded":
                lens = torch.tensor(_lengths(case["batch"], n, seed, max(1, n // 4)), device=DEVICE)
                s["pad"] = (torch.arange(n, device=DEVICE)[None] < lens[:, None]).long()
                s["mask"] = KeyPaddingMask(s["pad"])         # as ``BertModel`` makes it, once for all of its blocks
            if kind == "decoder":
                s["enc"] = rng.normal((case["batch"], case["enc"], hidden), 1.0).requires_grad_(True)
                dec = torch.tensor(_lengths(case["batch"], n, seed, max(1, n // 4)), device=DEVICE)
                enc = torch.tensor(_lengths(case["batch"], case["enc"], seed + 1, max(1, case["enc"] // 4)), device=DEVICE)
                pos, epos = torch.arange(n, device=DEVICE), torch.arange(case["enc"], device=DEVICE)
                q, k = pos[None] < dec[:, None], epos[None] < enc[:, None]
                s["mask"] = (q[:, :, None] & q[:, None, :] & (pos[None] <= pos[:, None])[None]).unsqueeze(1)   # as the T5 data set makes them
                s["cross_mask"] = (q[:, :, None] & k[:, None, :]).unsqueeze(1)
            return s
        if kind == "attend":
            s["qkv"] = rng.normal((case["batch"], case["seq"], case["heads"], 3 * case["dim"]), 1.0).requires_grad_(True)
            s["go"] = rng.normal((case["batch"], case["seq"], case["heads"], case["dim"]), 1.0)
            return s
        if kind == "head":
            emb = VocabEmbedding(case["vocab"], case["hidden"])
            _weights(rng, emb)
            s["emb"], s["head"], s["loss"], s["opt"] = emb, LMLogits(case["vocab"]), ParallelCrossEntropyLoss(), _optimizer(emb)
            s["x"] = rng.normal((case["batch"], case["seq"], case["hidden"]), 1.0).requires_grad_(True)
            s["labels"] = rng.ints((case["batch"], case["seq"]), case["vocab"])
            return s
        if kind == "adamw":
            blocks = torch.nn.ModuleList([_layer(case) for _ in range(case["layers"])])
            _weights(rng, blocks)
            s["opt"], s["params"] = _optimizer(blocks), list(blocks.parameters())
            for p in s["params"]:
                p.main_grad.copy_(rng.normal(p.shape, 1e-3, torch.float32))
            return s
        if kind == "gpt":
            model = s["model"] = GPTModel(DictConfig(dict(
                hidden_layers=case["layers"], vocab_size=case["vocab"], hidden_size=case["heads"] * case["dim"],
                ffn_hidden_size=case["ffn"], num_attention_heads=case["heads"], max_seq_length=1024, embedding_dropout_prob=0.0,
                attention_dropout_prob=0.0, output_dropout_prob=0.0, layernorm_epsilon=1e-5, initializer_range=0.02,
                use_scaled_init_for_output_weights=True, bias_gelu_fusion=True, bias_dropout_fusion=True,
                scale_mask_softmax_fusion=True, apply_query_key_layer_scaling=True, apply_residual_post_layernorm=False,
                amp_enabled=False))).eval()
            _weights(rng, model)
            s["ids"] = rng.ints((case["batch"], case["seq"]), case["vocab"])
            return s
        mixer = s["mixer"] = GatedDeltaMixer(case["width"], case["heads"], case["kv_heads"], case["dim"], case["dim"], 4)
        with torch.no_grad():
            for name, p in mixer.named_parameters():
                std, mean = (0.3, 0.0) if name.endswith("conv") else (0.1, 1.0) if name == "norm" else (0.5, 0.0) if p.dim() == 1 else (0.02, 0.0)
                p.copy_(rng.normal(p.shape, std, mean=mean))
        lens = s["lens"] = _lengths(case["sequences"], case["longest"], 0, max(1, case["longest"] // 4))   # shapes do not depend on the seed
        s["h"] = rng.normal((sum(lens), case["width"]), 1.0)
        channels = 2 * case["kv_heads"] * case["dim"] + case["heads"] * case["dim"]
        s["bufs"] = {"S": torch.zeros(len(lens), case["heads"], case["dim"], case["dim"], device=DEVICE),
                     "tail": torch.zeros(len(lens), 3, channels, dtype=BF16, device=DEVICE)}
        s["rb"] = RaggedBatch(lens, list(range(len(lens))), [0] * len(lens), DEVICE)
        return s


# -------------------------------------------------------------------------------------------------------------------- run
def run(s):
    kind = s["case"]["kind"]
    if kind == "decode":
        with torch.no_grad():
            if s["case"]["model"] == "llama":
                y, kv = s["layer"](s["x"], past_key_value=s["past"], cos_cached=s["cos"], sin_cached=s["sin"], use_cache=True)
            else:
                y, kv = s["layer"](s["x"], past_key_value=s["past"], use_cache=True)
        return [y, kv[0], kv[1]]
    if kind in ("block", "decoder", "llama"):
        s["opt"].zero_grad()
        s["x"].grad = None
        if kind == "llama":
            y = s["layer"](s["x"], cos_cached=s["cos"], sin_cached=s["sin"])
        elif kind == "decoder":
            s["enc"].grad = None
            y = s["layer"](s["x"], s["mask"], s["enc"], s["cross_mask"])
        else:
            y = s["layer"](s["x"], s.get("mask"))
        y.backward(s["gy"])
        s["opt"].sync_gradients()
        out = {"y": y, "dx": s["x"].grad, "dw": {name: p.main_grad for name, p in s["params"].items()}}
        if kind == "decoder":
            out["denc"] = s["enc"].grad
        return out
    if kind == "attend":
        s["qkv"].grad = None
        o = OF.attention_qkvpacked(s["qkv"], causal=s["case"]["causal"], scale=s["case"]["dim"] ** -0.5)
        o.backward(s["go"])
        return [o, s["qkv"].grad]
    if kind == "head":
        s["opt"].zero_grad()
        s["x"].grad = None
        w = s["emb"].weight
        loss = s["loss"](s["head"](s["x"], w), s["labels"])
        loss.mean().backward()
        s["opt"].sync_gradients()
        return [loss, s["x"].grad, w.main_grad]
    if kind == "adamw":
        s["opt"].step()
        flat = [g for g in s["opt"]._groups if g is not None]
        return {"params": s["params"], "norm": s["opt"].last_grad_norm,
                "state": [[g.master, g.state["exp_avg"], g.state["exp_avg_sq"]] for g in flat]}
    if kind == "gpt":
        with torch.no_grad():
            return s["model"](s["ids"])
    with torch.no_grad():
        y = s["mixer"](s["h"], s["rb"], s["bufs"])
    return [y, s["bufs"]["S"], s["bufs"]["tail"]]


# ------------------------------------------------------------------------------------------------------------------- work
def work(case):
    kind = case["kind"]
    if kind == "attend":
        n = case["batch"] * case["seq"] * case["heads"] * case["dim"]
        pairs = case["batch"] * case["heads"] * case["seq"] * ((case["seq"] + 1) / 2 if case["causal"] else case["seq"])
        return {"bytes": 2 * n * (3 + 1 + 1 + 3), "flops": 2 * case["dim"] * pairs * (2 + 4)}
    if kind == "head":
        t, h, v = case["batch"] * case["seq"], case["hidden"], case["vocab"]
        return {"bytes": 2 * v * h + 4 * v * h + 2 * 2 * t * h + 12 * t, "flops": 6 * t * h * v}
    if kind == "delta":
        t, w, hd, kd = case["sequences"] * case["longest"] * 0.625, case["width"], case["heads"] * case["dim"], case["kv_heads"] * case["dim"]
        mats = w * (2 * kd + 2 * hd + 2 * case["heads"]) + hd * w
        return {"bytes": 2 * mats + 4 * t * w + 4 * case["sequences"] * hd * case["dim"], "flops": 2 * t * mats + 6 * t * hd * case["dim"]}
    hidden = case["heads"] * case["dim"]
    llama = kind == "llama" or case.get("model") == "llama"
    mats = 4 * hidden * hidden + (3 if llama else 2) * hidden * case["ffn"]
    if kind == "adamw":
        n = case["layers"] * mats
        return {"bytes": n * (4 + 3 * 8 + 2), "flops": 16 * n}
    if kind == "gpt":
        t, emb = case["batch"] * case["seq"], case["vocab"] * hidden
        return {"bytes": 2 * (case["layers"] * mats + emb + t * case["vocab"]),
                "flops": 2 * t * (case["layers"] * mats + emb) + 2 * case["layers"] * t * case["seq"] * hidden}
    if kind == "decode":
        kv = 2 * case["batch"] * hidden
        return {"bytes": 2 * (mats + kv * case["past"] + kv * (case["past"] + 1) + 2 * case["batch"] * hidden),
                "flops": 2 * case["batch"] * mats + 4 * case["batch"] * hidden * (case["past"] + 1)}
    t = case["batch"] * case["seq"]
    pairs = t * case["seq"] * (0.5 if case.get("mask") == "causal" or kind == "llama" else 1.0)
    flops, more = 6 * t * mats + 12 * pairs * hidden, 0
    if kind == "decoder":
        enc = case["batch"] * case["enc"]
        mats += 4 * hidden * hidden
        flops = 6 * t * mats + 12 * enc * hidden * hidden - 12 * t * hidden * hidden + 12 * hidden * (0.5 * t * case["seq"] + t * case["enc"])
        more = 4 * enc * hidden
    return {"bytes": mats * (2 + 4) + 2 * t * hidden * 4 + more, "flops": flops}


def tolerance(case):
    # Relative errors against the 64-bit answer, measured, times about four.  Activations and gradients pass through bf16 at every
    # operator (2^-9 each), weight gradients and the optimizer's state are sums in 32 bits.
    if case["kind"] == "adamw":
        return {"rel": 2e-5, "max": 2e-2}          # one step of bf16 in a parameter now and then, fp32 sums everywhere else
    return {"rel": {"attend": 0.01, "head": 0.008, "llama": 0.03, "gpt": 0.028}.get(case["kind"], 0.02)}


# ------------------------------------------------------------------------------------------------------- 64-bit arithmetic
def _f64(t):
    return t.detach().to(torch.float64)


def _attend(q, k, v, scale, keep=None):
    """Softmax attention on ``[b, a, s, d]``, one sequence at a time; ``keep`` ``[b, 1, sq, sk]``: scores elsewhere are -10000."""
    out = []
    for i in range(q.shape[0]):
        w = q[i] @ k[i].transpose(-1, -2) * scale
        if keep is not None:
            w = torch.where(keep[i if keep.shape[0] > 1 else 0], w, torch.full_like(w, -10000.0))
        out.append(torch.softmax(w, -1) @ v[i])
    return torch.stack(out)


def _heads(x, heads):
    return x.view(x.shape[0], x.shape[1], heads, -1).permute(0, 2, 1, 3)


def _merge(x):
    return x.permute(0, 2, 1, 3).reshape(x.shape[0], x.shape[2], -1)


def _gelu(x):
    return 0.5 * x * (1.0 + torch.erf(x / math.sqrt(2.0)))


def _norm(x, w, b=None, eps=1e-5):
    if b is None:
        return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps) * w
    m = x.mean(-1, keepdim=True)
    return (x - m) * torch.rsqrt((x - m).square().mean(-1, keepdim=True) + eps) * w + b


def _block(p, x, heads, keep=None, enc=None, cross=None, past=None):
    """Pre-norm block from its parameters by name; returns the output and the keys and values."""
    lin = lambda name, v: v @ p[name + ".weight"].t() + p[name + ".bias"]
    norm = lambda name, v: _norm(v, p[name + ".weight"], p[name + ".bias"])
    dim = x.shape[-1] // heads
    q, k, v = _heads(lin("self_attention.query_key_value", norm("input_layernorm", x)), heads).split(dim, -1)
    if past is not None:
        k, v = torch.cat([past[0], k], 2), torch.cat([past[1], v], 2)
    x = x + lin("self_attention.dense", _merge(_attend(q, k, v, dim ** -0.5, keep)))
    h = norm("post_attention_layernorm", x)
    if enc is not None:
        ck, cv = _heads(lin("cross_attention.key_value", enc), heads).split(dim, -1)
        x = x + lin("cross_attention.dense", _merge(_attend(_heads(lin("cross_attention.query", h), heads), ck, cv, dim ** -0.5, cross)))
        h = norm("post_cross_attention_layernorm", x)
    return x + lin("mlp.dense_4h_to_h", _gelu(lin("mlp.dense_h_to_4h", h))), k, v


def _rotate(x, cos, sin):
    a, b = x.chunk(2, -1)
    return x * cos + torch.cat([-b, a], -1) * sin


def _llama(p, x, heads, cos, sin, past=None):
    dim, n = x.shape[-1] // heads, x.shape[1]
    at = 0 if past is None else past[0].shape[2]
    norm = lambda name, v: _norm(v, p[name + ".weight"], eps=1e-6)
    q, k, v = _heads(norm("input_layernorm", x) @ p["self_attn.query_key_value.weight"].t(), heads).split(dim, -1)
    q, k = _rotate(q, cos[at:at + n], sin[at:at + n]), _rotate(k, cos[at:at + n], sin[at:at + n])
    if past is not None:
        k, v = torch.cat([past[0], k], 2), torch.cat([past[1], v], 2)
    keep = None if past is not None else torch.ones(n, n, dtype=torch.bool, device=x.device).tril()[None, None]
    x = x + _merge(_attend(q, k, v, dim ** -0.5, keep)) @ p["self_attn.o_proj.weight"].t()
    h = norm("post_attention_layernorm", x)
    g = h @ p["mlp.gate_proj.weight"].t()
    return x + (g * torch.sigmoid(g) * (h @ p["mlp.up_proj.weight"].t())) @ p["mlp.down_proj.weight"].t(), k, v


def exact(case, seed):
    kind, s = case["kind"], prepare(case, seed)
    if kind == "adamw":
        groups = [(g, set(id(p) for p in g["params"])) for g in s["opt"].param_groups]
        total = math.sqrt(sum(float(_f64(p.main_grad).square().sum()) for p in s["params"]))
        coef, out = min(1.0, 1.0 / (total + 1e-6)), []
        for p in s["params"]:
            decay = next(g["weight_decay"] for g, ids in groups if id(p) in ids)
            g = _f64(p.main_grad) * coef
            m, v = 0.1 * g, 0.001 * g * g
            w = _f64(p)
            out.append(w - 1e-4 * (m / 0.1 / ((v / 0.001).sqrt() + 1e-8) + decay * w))
        return {"params": out, "norm": total, "state": None}
    if kind == "delta":
        return _exact_delta(case, s)
    if kind == "gpt":
        p = {n: _f64(t) for n, t in s["model"].named_parameters()}
        n = case["seq"]
        x = p["embeddings.token_embeddings.weight"][s["ids"]] + p["embeddings.position_embeddings.weight"][:n]
        keep = torch.ones(n, n, dtype=torch.bool, device=x.device).tril()[None, None]
        for i in range(case["layers"]):
            at = "transformer.layers.%d." % i
            x = _block({k[len(at):]: v for k, v in p.items() if k.startswith(at)}, x, case["heads"], keep)[0]
        x = _norm(x, p["transformer.layernorm_f.weight"], p["transformer.layernorm_f.bias"])
        return x @ p["embeddings.token_embeddings.weight"].t()
    if kind == "head":
        x, w = _f64(s["x"]).requires_grad_(True), _f64(s["emb"].weight).requires_grad_(True)
        z = (x @ w.t()).flatten(0, 1)
        loss = torch.nn.functional.cross_entropy(z, s["labels"].flatten(), reduction="none").view(s["labels"].shape)
        loss.mean().backward()
        return [loss, x.grad, w.grad]
    if kind == "attend":
        qkv, n = _f64(s["qkv"]).requires_grad_(True), case["seq"]
        keep = torch.ones(n, n, dtype=torch.bool, device=DEVICE).tril() if case["causal"] else None
        o = torch.empty(qkv.shape[0], n, case["heads"], case["dim"], dtype=torch.float64, device=DEVICE)
        for b in range(qkv.shape[0]):
            for a in range(case["heads"]):           # one head at a time: the scores of a long sequence are large in 64 bits
                q, k, v = qkv[b, :, a].split(case["dim"], -1)
                z = q @ k.t() * case["dim"] ** -0.5
                part = torch.softmax(z if keep is None else z.masked_fill(~keep, -math.inf), -1) @ v
                part.backward(_f64(s["go"][b, :, a]))
                o[b, :, a] = part.detach()
        return [o, qkv.grad]
    p = {n: _f64(t) for n, t in s["layer"].named_parameters()}
    if kind == "decode":
        past = tuple(_f64(t) for t in s["past"])
        if case["model"] == "llama":
            return list(_llama(p, _f64(s["x"]), case["heads"], _f64(s["cos"]), _f64(s["sin"]), past))
        return list(_block(p, _f64(s["x"]), case["heads"], past=past))
    for t in p.values():
        t.requires_grad_(True)
    x = _f64(s["x"]).requires_grad_(True)
    enc = None
    if kind == "llama":
        y = _llama(p, x, case["heads"], _f64(s["cos"]), _f64(s["sin"]))[0]
    elif kind == "decoder":
        enc = _f64(s["enc"]).requires_grad_(True)
        y = _block(p, x, case["heads"], s["mask"], enc, s["cross_mask"])[0]
    else:
        n, keep = case["seq"], None
        if case["mask"] == "causal":
            keep = torch.ones(n, n, dtype=torch.bool, device=DEVICE).tril()[None, None]
        elif case["mask"] == "padded":
            keep = s["pad"].bool()[:, None, None, :]
            if case["dim"] not in (64, 128):       # rows behind a sequence's end (nobody reads them): all scores alike there
                keep = keep & s["pad"].bool()[:, None, :, None]
        y = _block(p, x, case["heads"], keep)[0]
    y.backward(_f64(s["gy"]))
    out = {"y": y, "dx": x.grad, "dw": {n: t.grad for n, t in p.items()}}
    if enc is not None:
        out["denc"] = enc.grad
    return out


def _exact_delta(case, s):
    """The recurrence of the mixer, token by token, all sequences side by side."""
    p = {n: _f64(t) for n, t in s["mixer"].named_parameters()}
    lens, H, G, D = s["lens"], case["heads"], case["kv_heads"], case["dim"]
    n, B = max(lens), len(lens)
    h = torch.zeros(B, n + 3, case["width"], dtype=torch.float64, device=DEVICE)
    at = 0
    for i, m in enumerate(lens):
        h[i, 3:3 + m] = _f64(s["h"][at:at + m])
        at += m
    raw = h @ torch.cat([p["q"], p["k"], p["v"]]).t()
    taps = torch.cat([p["q_conv"], p["k_conv"], p["v_conv"]])
    conv = sum(raw[:, j:j + n] * taps[:, j] for j in range(4))
    conv = conv * torch.sigmoid(conv)
    q, k, v = conv.split([G * D, G * D, H * D], -1)
    unit = lambda t: t / torch.sqrt(t.square().sum(-1, keepdim=True) + 1e-6)
    q = unit(q.view(B, n, G, D)).repeat_interleave(H // G, 2) / math.sqrt(D)
    k, v = unit(k.view(B, n, G, D)).repeat_interleave(H // G, 2), v.view(B, n, H, D)
    x = h[:, 3:]
    beta = torch.sigmoid(x @ p["b"].t())
    decay = torch.exp(-torch.exp(p["A_log"]) * torch.nn.functional.softplus(x @ p["a"].t() + p["dt_bias"], threshold=200.0))
    state = torch.zeros(B, H, D, D, dtype=torch.float64, device=DEVICE)
    live = torch.arange(n, device=DEVICE)[:, None] < torch.tensor(lens, device=DEVICE)[None]
    outs = []
    for t in range(n):
        new = state * decay[:, t, :, None, None]
        u = beta[:, t, :, None] * (v[:, t] - torch.einsum("bhdv,bhd->bhv", new, k[:, t]))
        new = new + k[:, t, :, :, None] * u[:, :, None, :]
        state = torch.where(live[t][:, None, None, None], new, state)
        outs.append(torch.einsum("bhdv,bhd->bhv", new, q[:, t]))
    o = torch.stack(outs, 1)
    o = o * torch.rsqrt(o.square().mean(-1, keepdim=True) + 1e-6) * p["norm"]
    g = (x @ p["g"].t()).view(B, n, H, D)
    y = (o * g * torch.sigmoid(g)).reshape(B, n, H * D) @ p["o"].t()
    tail = torch.stack([raw[i, m:m + 3] for i, m in enumerate(lens)])
    return [torch.cat([y[i, :m] for i, m in enumerate(lens)]), state, tail]
