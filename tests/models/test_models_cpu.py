"""Every model family builds from its packaged config, runs forward + backward on CPU and produces finite losses and
gradients for all parameters (the reference's per-model tests need GPUs + downloaded corpora; these are the CPU
counterpart on synthetic batches — the multi-rank layout equivalence lives in tests/test_parallel_cpu.py)."""
import pytest
import torch

from libai_b200.config import LazyConfig, instantiate

NLP_OVERRIDES = ["model.cfg.hidden_size=48", "model.cfg.num_attention_heads=4", "model.cfg.hidden_layers=2",
                 "model.cfg.vocab_size=128"]


def _check(model, out_loss):
    assert torch.isfinite(out_loss).all()
    out_loss.backward()
    missing = [n for n, p in model.named_parameters() if p.requires_grad and p.grad is None
               and getattr(p, "main_grad", None) is None]
    assert not missing, missing


def _load(cfg_file, overrides):
    cfg = LazyConfig.load(cfg_file)
    return LazyConfig.apply_overrides(cfg, overrides)


def test_gpt():
    cfg = _load("configs/gpt2_pretrain.py", NLP_OVERRIDES + ["model.cfg.ffn_hidden_size=96", "model.cfg.max_seq_length=32"])
    model = instantiate(cfg.model).train()
    ids = torch.randint(0, 128, (2, 32))
    out = model(ids, ids)
    assert set(out) == {"lm_loss"}
    _check(model, out["lm_loss"])
    model.eval()
    assert model(ids)["prediction_scores"].shape == (2, 32, 128)


def test_bert_pretraining_and_classification():
    cfg = _load("configs/bert_large_pretrain.py", NLP_OVERRIDES + ["model.cfg.intermediate_size=96", "model.cfg.max_position_embeddings=32"])
    model = instantiate(cfg.model).train()
    ids = torch.randint(0, 128, (2, 32))
    mask = torch.ones(2, 32, dtype=torch.long)
    mask[1, 20:] = 0
    out = model(ids, mask, torch.zeros_like(ids), ns_labels=torch.tensor([0, 1]), lm_labels=ids, loss_mask=mask)
    assert {"lm_loss", "sop_loss"} <= set(out)
    _check(model, out["lm_loss"] + out["sop_loss"])
    cfg = _load("configs/bert_classification.py", NLP_OVERRIDES + ["model.cfg.intermediate_size=96", "model.cfg.max_position_embeddings=32"])
    clf = instantiate(cfg.model).train()
    out = clf(ids, mask, torch.zeros_like(ids), labels=torch.tensor([0, 1]))
    _check(clf, out["loss"] if "loss" in out else next(iter(out.values())))


def test_roberta():
    cfg = _load("configs/roberta_pretrain.py", NLP_OVERRIDES + ["model.cfg.intermediate_size=96", "model.cfg.max_position_embeddings=40"])
    model = instantiate(cfg.model).train()
    ids = torch.randint(2, 128, (2, 32))
    mask = torch.ones(2, 32, dtype=torch.long)
    out = model(ids, mask, torch.zeros_like(ids), lm_labels=ids, loss_mask=mask)
    _check(model, out["lm_loss"])


def test_t5():
    cfg = _load("configs/t5_large_pretrain.py", NLP_OVERRIDES + ["model.cfg.intermediate_size=96", "model.cfg.max_position_embeddings=32"])
    model = instantiate(cfg.model).train()
    enc, dec = torch.randint(0, 128, (2, 16)), torch.randint(0, 128, (2, 8))
    out = model(enc, dec, torch.ones(2, 16, 16, dtype=torch.bool), torch.ones(2, 8, 8, dtype=torch.bool).tril(),
                torch.ones(2, 8, 16, dtype=torch.bool), lm_labels=dec, loss_mask=torch.ones(2, 8))
    _check(model, out["masked_lm_loss"])


def test_llama():
    cfg = LazyConfig.load("configs/common/models/llama.py")
    cfg = LazyConfig.apply_overrides(cfg, ["cfg.hidden_layers=2", "cfg.hidden_size=64", "cfg.intermediate_size=128",
                                           "cfg.num_attention_heads=4", "cfg.vocab_size=128", "cfg.max_position_embeddings=32"])
    cfg.model.cfg = cfg.cfg
    model = instantiate(cfg.model).train()
    ids = torch.randint(1, 128, (2, 16))
    _check(model, model(ids, labels=ids)["lm_loss"])


@pytest.mark.parametrize("recipe,overrides,size", [
    ("configs/vit_imagenet.py", ["model.cfg.embed_dim=48", "model.cfg.depth=2", "model.cfg.num_heads=4", "model.cfg.img_size=32", "model.cfg.patch_size=8"], 32),
    ("configs/swin_imagenet.py", ["model.cfg.embed_dim=16", "model.cfg.depths=[2,2]", "model.cfg.num_heads=[2,4]", "model.cfg.img_size=32", "model.cfg.patch_size=2", "model.cfg.window_size=4"], 32),
    ("configs/swinv2_imagenet.py", ["model.cfg.embed_dim=16", "model.cfg.depths=[2,2]", "model.cfg.num_heads=[2,4]", "model.cfg.img_size=32", "model.cfg.patch_size=2", "model.cfg.window_size=4", "model.cfg.pretrained_window_sizes=[0,0]"], 32),
    ("configs/resmlp_imagenet.py", ["model.cfg.embed_dim=48", "model.cfg.depth=2", "model.cfg.img_size=32", "model.cfg.patch_size=8"], 32),
])
def test_vision_models_with_mixup(recipe, overrides, size):
    cfg = _load(recipe, overrides + ["model.cfg.num_classes=10", "dataloader.train.mixup_func.num_classes=10"])
    model = instantiate(cfg.model).train()
    mixup = instantiate(cfg.dataloader.train.mixup_func)
    images, soft = mixup(torch.randn(4, 3, size, size), torch.tensor([1, 2, 3, 4]))
    out = model(images, soft)
    _check(model, out["losses"])
    model.eval()
    assert model(images)["prediction_scores"].shape == (4, 10)


def _small_block(kind, dtype):
    from libai_b200.layers import TransformerLayer
    from libai_b200.layers._param import param_defaults
    from libai_b200.models.llama_model import LlamaDecoderLayer, rotary_tables

    with param_defaults(dtype=dtype, seed=5):
        m = LlamaDecoderLayer(32, 64, 4) if kind == "llama" else TransformerLayer(32, 64, 4)
    tables = dict(zip(("cos_cached", "sin_cached"), rotary_tables(8, 16))) if kind == "llama" else {}
    x = torch.randn(2, 6, 32, generator=torch.Generator().manual_seed(1)).to(dtype).requires_grad_(True)
    return m, x, lambda: m(x, **tables)


# what a block calls as modules (the GPT block's norms and, in bf16, its projections have always been joined with their neighbours)
SEEN = {"llama": {"input_layernorm", "self_attn", "self_attn.query_key_value", "self_attn.o_proj", "post_attention_layernorm", "mlp", "mlp.gate_proj",
                  "mlp.up_proj", "mlp.down_proj"},
        "gpt": {"self_attention", "self_attention.query_key_value", "self_attention.dense", "mlp"}}


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("kind", ["llama", "gpt"])
@pytest.mark.parametrize("how", ["backward", "backward_pre", "global_forward", "global_forward_pre", "global_backward"])
def test_hooks_see_the_modules_of_a_block(kind, how, dtype):
    """Residual adds in epilogues and skip gradients in the norms' backward pass modules by: not while anything looks at their calls."""
    from torch.nn.modules import module as hooks

    m, x, call = _small_block(kind, dtype)
    names, seen, handles = {k: n for n, k in m.named_modules()}, set(), []
    note = lambda mod, *a: seen.add(names[mod])
    if how.startswith("global"):
        register = {"global_forward": hooks.register_module_forward_hook, "global_forward_pre": hooks.register_module_forward_pre_hook,
                    "global_backward": hooks.register_module_full_backward_hook}[how]
        handles.append(register(note))
    else:
        for n, k in m.named_modules():
            if n:
                handles.append(k.register_full_backward_hook(note) if how == "backward" else k.register_full_backward_pre_hook(note))
    try:
        call().sum().backward()
    finally:
        for h in handles:
            h.remove()
    joined = {"self_attention.dense"} if kind == "gpt" and dtype == torch.bfloat16 else set()
    assert seen - {""} == SEEN[kind] - joined


@pytest.mark.parametrize("name", ["input_layernorm", "post_attention_layernorm", "self_attn", "self_attn.o_proj", "mlp", "mlp.down_proj"])
def test_backward_hooks_of_a_llama_block_change_their_branch_only(name):
    """A hook that drops the gradient at a module's output drops that branch and keeps the skip connection."""
    m, x, call = _small_block("llama", torch.bfloat16)
    whole = torch.autograd.grad(call().sum(), x)[0]
    h = m.get_submodule(name).register_full_backward_pre_hook(lambda mod, gy: tuple(torch.zeros_like(g) for g in gy))
    cut = torch.autograd.grad(call().sum(), x)[0]
    h.remove()
    branch = m.self_attn if name in ("input_layernorm", "self_attn", "self_attn.o_proj") else m.mlp
    forward = branch.forward
    branch.forward = lambda *a, **k: forward(*a, **k).detach()               # the same by hand
    want = torch.autograd.grad(call().sum(), x)[0]
    assert torch.equal(cut, want) and not torch.equal(cut, whole)


def test_modules_with_another_call_are_not_passed_by(monkeypatch):
    from libai_b200.layers import RMSLayerNorm
    from libai_b200.layers import _native_block as native

    m = _small_block("llama", torch.float32)[0].input_layernorm
    assert native.alone(m, RMSLayerNorm)
    call = torch.nn.Module.__call__
    with monkeypatch.context() as patch:                      # as tracers and profilers do
        patch.setattr(torch.nn.Module, "__call__", lambda self, *a, **k: call(self, *a, **k))
        assert not native.alone(m, RMSLayerNorm)
    assert native.alone(m, RMSLayerNorm)
    m.compile(backend="eager")
    assert not native.plain(m, RMSLayerNorm)
