"""One transformer block (encoder or decoder flavour).

Spec: reference libai/layers/transformer_layer.py:26-248 — pre-LN by default
(``apply_residual_post_layernorm`` takes the residual *after* the LN instead), optional
cross-attention for decoders, DropPath on both residual branches, KV cache passthrough.
The pipeline hand-off the reference performs inside ``forward`` (``to_global(placement=…)``,
:158) is done by the pipeline engine between stages, not here.
"""
from torch import nn

from libai_b200.ops import functional as OF, fused_bias_grad, load_ext

from . import _native_block as native
from ._param import xavier_normal_
from .attention import AttnMaskType, KeyPaddingMask, MultiheadAttention
from .droppath import DropPath
from .layer_norm import LayerNorm
from .linear import Linear
from .mlp import MLP

native.remember(LayerNorm, MultiheadAttention, Linear, MLP)


class TransformerLayer(nn.Module):
    def __init__(
        self,
        hidden_size,
        ffn_hidden_size,
        num_attention_heads,
        is_decoder=False,
        attention_dropout_prob=0.0,
        output_dropout_prob=0.0,
        drop_path_prob=0.0,
        layernorm_epsilon=1e-5,
        init_method=xavier_normal_,
        output_layer_init_method=None,
        bias_gelu_fusion=False,
        bias_dropout_fusion=False,
        scale_mask_softmax_fusion=False,
        apply_query_key_layer_scaling=False,
        apply_residual_post_layernorm=False,
        attn_mask_type=AttnMaskType.padding,
        *,
        layer_idx=0,
    ):
        super().__init__()
        self.hidden_size = hidden_size
        self.ffn_hidden_size = ffn_hidden_size
        self.num_attention_heads = num_attention_heads
        self.attention_dropout_prob = attention_dropout_prob
        self.output_dropout_prob = output_dropout_prob
        self.layernorm_epsilon = layernorm_epsilon
        self.attn_mask_type = attn_mask_type
        self.layer_idx = layer_idx
        self.is_decoder = is_decoder
        self.bias_gelu_fusion = bias_gelu_fusion
        self.bias_dropout_fusion = bias_dropout_fusion
        self.scale_mask_softmax_fusion = scale_mask_softmax_fusion
        self.apply_query_key_layer_scaling = apply_query_key_layer_scaling
        self.apply_residual_post_layernorm = apply_residual_post_layernorm
        self.init_method = init_method
        self.output_layer_init_method = output_layer_init_method or init_method
        self.drop_path = DropPath(drop_path_prob) if drop_path_prob > 0.0 else nn.Identity()
        self.plain_residual = drop_path_prob == 0.0

        self.input_layernorm = LayerNorm(hidden_size, eps=layernorm_epsilon, layer_idx=layer_idx)
        self.self_attention = self.build_attention(is_cross_attention=False)
        self.post_attention_layernorm = LayerNorm(hidden_size, eps=layernorm_epsilon, layer_idx=layer_idx)
        if self.is_decoder:
            self.cross_attention = self.build_attention(is_cross_attention=True)
            self.post_cross_attention_layernorm = LayerNorm(hidden_size, eps=layernorm_epsilon, layer_idx=layer_idx)
        self.mlp = MLP(
            hidden_size, ffn_hidden_size, output_dropout_prob, init_method,
            output_layer_init_method=self.output_layer_init_method,
            bias_gelu_fusion=bias_gelu_fusion, bias_dropout_fusion=bias_dropout_fusion, layer_idx=layer_idx,
        )

    def _branch(self, fn, residual, **kw):
        """residual + drop_path(fn(...)); the add is fused into fn's epilogue when no DropPath."""
        if self.plain_residual:
            return fn(residual=residual, **kw)
        out = fn(residual=None, **kw)
        if isinstance(out, tuple):
            return (residual + self.drop_path(out[0]),) + tuple(out[1:])
        return residual + self.drop_path(out)

    def forward(
        self,
        hidden_states,
        attention_mask=None,
        encoder_states=None,
        encoder_attention_mask=None,
        past_key_value=None,
        use_cache=False,
    ):
        """``past_key_value``: ``(self_k, self_v[, cross_k, cross_v])``; returns hidden states, and
        the updated cache tuple when ``use_cache``."""
        if attention_mask is None and encoder_states is None and native.applies(hidden_states):
            done = self._native_forward(hidden_states, past_key_value, use_cache)
            if done is not None:
                return done
        elif past_key_value is None and not use_cache and native.applies_with_graph(hidden_states):
            done = self._graph_forward(hidden_states, attention_mask, encoder_states, encoder_attention_mask)
            if done is not None:
                return done
        self_past = cross_past = None
        if past_key_value is not None:
            self_past = past_key_value[:2]
            cross_past = past_key_value[2:] if len(past_key_value) > 2 else None
            cross_past = cross_past or None

        if self.apply_residual_post_layernorm:
            ln = self.input_layernorm(hidden_states)
            residual = ln
        else:   # pre-LN: the skip gradient is folded into the LayerNorm backward kernel
            ln, residual = self.input_layernorm.forward_with_skip(hidden_states)
        attn = self._branch(
            lambda residual, **kw: self.self_attention(ln, residual=residual, **kw),
            residual, attention_mask=attention_mask, past_key_value=self_past, use_cache=use_cache,
        )
        presents = None
        if use_cache:
            attn, presents = attn
        hidden_states = attn

        if self.apply_residual_post_layernorm or self.is_decoder:
            ln = self.post_attention_layernorm(hidden_states)
            post_skip = hidden_states
        else:
            ln, post_skip = self.post_attention_layernorm.forward_with_skip(hidden_states)
        if self.is_decoder:
            residual = ln if self.apply_residual_post_layernorm else hidden_states
            cross = self._branch(
                lambda residual, **kw: self.cross_attention(ln, residual=residual, **kw),
                residual, encoder_states=encoder_states, attention_mask=encoder_attention_mask,
                past_key_value=cross_past, use_cache=use_cache,
            )
            if use_cache:
                cross, cross_kv = cross
                presents = tuple(presents) + tuple(cross_kv)
            hidden_states = cross
            ln = self.post_cross_attention_layernorm(hidden_states)
            residual = ln if self.apply_residual_post_layernorm else hidden_states
        elif self.apply_residual_post_layernorm:
            residual = ln
        else:
            residual = post_skip
        output = self._branch(lambda residual: self.mlp(ln, residual=residual), residual)
        if use_cache:
            return output, presents
        return output

    def _native_forward(self, x, past, use_cache):
        """The block without a graph as one native call; ``None``: the modules have to run."""
        if self.is_decoder or self.apply_residual_post_layernorm or not self.plain_residual or (use_cache and past is None):
            return None
        mods = self._modules
        ln1, attn, ln2, mlp = mods["input_layernorm"], mods["self_attention"], mods["post_attention_layernorm"], mods["mlp"]
        plain = native.plain
        if not (plain(ln1, LayerNorm) and plain(attn, MultiheadAttention) and plain(ln2, LayerNorm) and plain(mlp, MLP)):
            return None
        qkv, dense, up, down = attn._modules.get("query_key_value"), attn._modules["dense"], mlp._modules["dense_h_to_4h"], mlp._modules["dense_4h_to_h"]
        if (not (plain(qkv, Linear) and plain(dense, Linear) and plain(up, Linear) and plain(down, Linear))
                or qkv.skip_bias_add or up.skip_bias_add or len(ln1.normalized_shape) != 1 or len(ln2.normalized_shape) != 1
                or (attn.training and (attn.attention_dropout_prob > 0.0 or attn.output_dropout_prob > 0.0)) or (mlp.training and mlp.output_dropout_prob > 0.0)):
            return None
        both = ("weight", "bias")
        params = native.parameters((ln1, *both), (qkv, *both), (dense, *both), (ln2, *both), (up, *both), (down, *both))
        pair = native.past_pair(past, attn.local_heads, x)
        if params is None or pair is None:
            return None
        out = load_ext().block_fwd(x, params, attn.local_heads, ln1.eps, ln2.eps, attn.softmax_scale, attn.attn_mask_type == AttnMaskType.causal, *pair)
        if not out:
            return None
        return (out[0], tuple(out[1:])) if use_cache else out[0]

    def _graph_forward(self, x, mask, enc, cross_mask):
        """The block's graph as one native call; ``None``: the modules have to run."""
        if self.apply_residual_post_layernorm or not self.plain_residual or self.is_decoder != (enc is not None):
            return None
        mods = self._modules
        plain = native.plain_with_graph
        attn, mlp = mods["self_attention"], mods["mlp"]
        if not (plain(attn, MultiheadAttention) and plain(mlp, MLP)) or (mlp.training and mlp.output_dropout_prob > 0.0):
            return None
        parts = [(mods["input_layernorm"], LayerNorm), (attn._modules.get("query_key_value"), Linear), (attn._modules["dense"], Linear)]
        cross = None
        if enc is not None:
            cross = mods["cross_attention"]
            if not plain(cross, MultiheadAttention) or not OF._graph_node(enc) or enc.dim() != 3 or cross.local_heads != attn.local_heads:
                return None
            parts += [(mods["post_attention_layernorm"], LayerNorm), (cross._modules.get("query"), Linear), (cross._modules.get("key_value"), Linear),
                      (cross._modules["dense"], Linear), (mods["post_cross_attention_layernorm"], LayerNorm)]
        else:
            parts.append((mods["post_attention_layernorm"], LayerNorm))
        parts += [(mlp._modules["dense_h_to_4h"], Linear), (mlp._modules["dense_4h_to_h"], Linear)]
        for m, cls in parts:
            if m is None or not plain(m, cls) or (cls is LayerNorm and len(m.normalized_shape) != 1):
                return None
        if attn._modules["query_key_value"].skip_bias_add or mlp._modules["dense_h_to_4h"].skip_bias_add:
            return None
        for a in (attn, cross):
            if a is not None and a.training and (a.attention_dropout_prob > 0.0 or a.output_dropout_prob > 0.0):
                return None
        params = native.parameters(*((m, "weight", "bias") for m, _ in parts))
        if params is None:
            return None
        # the kernels that ``MultiheadAttention.forward`` would pick: flash (head dims 64 and 128, lengths of a right-padded batch) or with 32-bit probabilities
        (b, s, _), heads, d, lens = x.shape, attn.local_heads, attn.head_size, None
        causal = attn.attn_mask_type == AttnMaskType.causal
        if isinstance(mask, KeyPaddingMask):
            if d in (64, 128) and mask.is_prefix():
                mask, lens = None, mask.lengths
            else:
                mask = mask.dense()
        if ((mask is not None or d not in (64, 128)) and not self._split_attention_takes(x, mask, (b, heads, s), s, d, attn.softmax_scale, causal and mask is None)
                or not OF._graph_node(mask, lens)):
            return None
        if cross is not None:
            if isinstance(cross_mask, KeyPaddingMask):
                cross_mask = cross_mask.dense()
            if not self._split_attention_takes(x, cross_mask, (b, heads, s), enc.shape[1], cross.head_size, cross.softmax_scale, False) or not OF._graph_node(cross_mask):
                return None
        out = load_ext().block_nodes(x, params, heads, [m.eps for m, cls in parts if cls is LayerNorm], float(attn.softmax_scale), causal, lens, mask, enc, cross_mask,
                                     0.0 if cross is None else float(cross.softmax_scale), fused_bias_grad())
        return out[0] if out else None

    @staticmethod
    def _split_attention_takes(x, mask, q_sizes, keys, d, scale, causal):
        return OF._split_sizes_ok(*q_sizes, keys, d, scale, causal) and (mask is None or OF._mask_supported(mask, q_sizes, x.device, keys))

    def build_attention(self, is_cross_attention=False):
        return MultiheadAttention(
            self.hidden_size, self.num_attention_heads,
            is_cross_attention=is_cross_attention,
            attention_dropout_prob=self.attention_dropout_prob,
            output_dropout_prob=self.output_dropout_prob,
            init_method=self.init_method, output_layer_init_method=self.output_layer_init_method,
            bias_dropout_fusion=self.bias_dropout_fusion,
            scale_mask_softmax_fusion=self.scale_mask_softmax_fusion,
            apply_query_key_layer_scaling=self.apply_query_key_layer_scaling,
            attn_mask_type=self.attn_mask_type, layer_idx=self.layer_idx,
        )
