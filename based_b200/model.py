"""Inference-only assembly of the Based language model on the B200 kernels.

Mirrors the module tree and parameter names of the reference's ``GPTLMHeadModel``
(based/models/gpt.py:737-830: ``transformer.embeddings.word_embeddings``, ``transformer.layers.N``
with ``mixer`` / ``norm1`` / ``mlp`` / ``norm2`` as in based/models/block.py:27-93,
``transformer.ln_f``, ``lm_head`` tied to the embedding, gpt.py:781-785), so a reference
checkpoint loads with ``load_state_dict``.  Only what generation needs is here: the prenorm
block of block.py:134-163 with an fp32 residual stream, layer selection by index as
``create_mixer_cls`` does it (gpt.py:64-96), greedy decoding with the prompt pass / single-token
steps split of based/generation.py:93-204, and optional CUDA-graph replay of the decode step
(:689-739).  Training, dropout, tensor-parallel embeddings and sampling strategies are not.
"""
from dataclasses import dataclass, field, fields
from typing import List, NamedTuple, Optional

import torch
import torch.nn as nn
import torch.nn.functional as F

from . import ops
from .generation import GenerationMixin, sample_token  # noqa: F401
from .mixers import BaseConv, LinearAttention, SlidingAttention, TaylorExp
from .modules import GatedMlp, RMSNorm


@dataclass
class BasedConfig:
    """The fields of the reference's experiment configs that shape the model
    (train/configs/experiment/reference/based-360m.yaml:49-117)."""
    n_embd: int = 1024
    n_layer: int = 27
    n_head: int = 16
    n_inner: Optional[int] = None              # GatedMlp hidden size; None -> 2 * n_embd as in the configs
    vocab_size: int = 50277
    pad_vocab_size_multiple: int = 8
    layer_norm_epsilon: float = 1e-5
    alt_mixer_layers: List[int] = field(default_factory=lambda: [1, 6, 11, 16, 21])      # LinearAttention
    alt_mixer_2_layers: List[int] = field(default_factory=lambda: [2, 7, 12, 17, 22])    # SlidingAttention
    conv_expand_proj: int = 4
    conv_kernel_size: int = 3
    feature_dim: int = 16
    window_size: int = 128                     # SlidingAttention window_size; the kernel window is window_size // 2
    rotary_emb_fraction: float = 1.0
    residual_in_fp32: bool = True
    l_max: int = 2048

    @property
    def padded_vocab_size(self):
        m = self.pad_vocab_size_multiple
        return (self.vocab_size + m - 1) // m * m

    @classmethod
    def from_dict(cls, d):
        """From the keys of a config file; keys that are not fields of this class are ignored."""
        return cls(**{f.name: d[f.name] for f in fields(cls) if f.name in d})

    @classmethod
    def based_360m(cls):
        return cls()

    @classmethod
    def based_1b(cls):
        """train/configs/experiment/reference/based-1b.yaml:50-123."""
        return cls(n_embd=1792, n_layer=36, alt_mixer_layers=[1, 6, 11, 16, 21, 27, 33],
                   alt_mixer_2_layers=[2, 7, 12, 17, 22, 28, 34])


_MIXERS = (BaseConv, LinearAttention, SlidingAttention)


class PromptPlan(NamedTuple):
    """What a prompt's pass through a layer without launches for the norms needs.  ``in_proj``, its bias and ``taps`` are a BaseConv layer's."""
    mixer: nn.Module
    norm1: RMSNorm
    norm2: RMSNorm
    fc1: torch.Tensor
    fc1_bias: Optional[torch.Tensor]
    fc2: torch.Tensor
    fc2_bias: Optional[torch.Tensor]
    activation: int
    out_proj: torch.Tensor
    out_bias: Optional[torch.Tensor]
    in_proj: Optional[torch.Tensor]
    in_bias: Optional[torch.Tensor]
    taps: Optional[torch.Tensor]
    norm1_weight: torch.Tensor
    norm2_weight: torch.Tensor


class Block(nn.Module):
    """Prenorm block: add -> norm -> mixer -> add -> norm -> MLP, returning (hidden, residual)."""

    def __init__(self, config: BasedConfig, layer_idx: int, device=None, dtype=None):
        super().__init__()
        fk = {"device": device, "dtype": dtype}
        d = config.n_embd
        self.layer_idx = layer_idx
        self.residual_in_fp32 = config.residual_in_fp32
        if layer_idx in config.alt_mixer_layers:
            self.mixer = LinearAttention(d, feature_map=TaylorExp(input_dim=config.feature_dim), l_max=config.l_max,
                                         feature_dim=config.feature_dim, num_heads=config.n_head, layer_idx=layer_idx,
                                         fuse_qkv=True, **fk)
        elif layer_idx in config.alt_mixer_2_layers:
            head_dim = d // config.n_head
            self.mixer = SlidingAttention(d, num_heads=config.n_head, window_size=config.window_size, causal=True,
                                          qkv_proj_bias=False, out_proj_bias=False, layer_idx=layer_idx,
                                          rotary_emb_dim=int(config.rotary_emb_fraction * head_dim), **fk)
        else:
            self.mixer = BaseConv(d, l_max=config.l_max, kernel_size=config.conv_kernel_size, layer_idx=layer_idx,
                                  use_bias=True, expand_proj=config.conv_expand_proj, **fk)
        self.norm1 = RMSNorm(d, eps=config.layer_norm_epsilon, **fk)
        self.mlp = GatedMlp(d, hidden_features=config.n_inner or 2 * d, activation=F.silu, bias1=False, bias2=False, **fk)
        self.norm2 = RMSNorm(d, eps=config.layer_norm_epsilon, **fk)

    def allocate_inference_cache(self, batch_size, max_seqlen, dtype=None, **kwargs):
        return self.mixer.allocate_inference_cache(batch_size, max_seqlen, dtype=dtype, **kwargs)

    def step_ok(self, width):
        """True when a decode step may run without launches of their own for the norms: the stream is fp32, nobody watches the
        modules or has put another forward on them, and the products around them are ones :func:`ops.linear_add_norm` and
        :func:`ops.decode_linear` take."""
        norms = (self.norm1, self.norm2)
        weights = self.mixer.step_weights() if type(self.mixer) in (BaseConv, LinearAttention, SlidingAttention) else None
        if weights is None or not self.residual_in_fp32 or type(self.mlp) is not GatedMlp or self.mlp.return_residual:
            return False
        if any(m._forward_hooks or m._forward_pre_hooks or "forward" in vars(m) for m in (self, self.mixer, self.mlp, *norms)):
            return False
        if any(type(n) is not RMSNorm or n.bias is not None or n.weight.dtype != torch.bfloat16 for n in norms):
            return False
        weights = weights + [(self.mlp.fc1.weight, self.mlp.fc1.bias), (self.mlp.fc2.weight, self.mlp.fc2.bias)]
        return (all(ops.step_weight(*w) for w in weights) and self.mlp.fc1.weight.shape[0] % 16 == 0
                and weights[-3][0].shape[0] == weights[-1][0].shape[0] == width)

    def prompt_plan(self, width):
        """This layer's :class:`PromptPlan`; None where :meth:`forward` has to run instead: somebody watches a module (hooks on all modules
        are the caller's to look for) or has put another forward on one, the stream is not fp32, or a module is not of the kind or form
        the kernels stand for.  Modules' own dictionaries are read, because a module's attribute look-up costs a microsecond and this
        runs for every layer of every prompt."""
        mods = self._modules
        mixer, mlp, norms = mods["mixer"], mods["mlp"], (mods["norm1"], mods["norm2"])
        kind, norm1, norm2 = type(mixer), *norms
        if kind not in _MIXERS or type(mlp) is not GatedMlp or not self.residual_in_fp32 or mlp.return_residual:
            return None
        if kind is LinearAttention and (not mixer.fuse_qkv or mixer.training) or kind is SlidingAttention and mixer.return_residual:
            return None
        if kind is not BaseConv and mixer.process_group is not None:
            return None
        fc1, fc2, out = mlp._modules["fc1"], mlp._modules["fc2"], mixer._modules["out_proj"]
        for m in (self, mixer, mlp, norm1, norm2, fc1, out):   # a prompt calls fc1 and out_proj as modules, too
            if m._forward_hooks or m._forward_pre_hooks or "forward" in m.__dict__:
                return None
        if "hidden" in mlp.__dict__ or "parallel_forward" in mixer.__dict__:
            return None
        act = 0 if mlp.activation is F.silu else 1 if mlp.activation in (F.sigmoid, torch.sigmoid) else None
        if act is None or type(fc1) is not nn.Linear or type(out) is not nn.Linear:
            return None
        own = []
        for m in norms:
            if type(m) is not RMSNorm or m._parameters.get("bias") is not None:
                return None
        for m in (fc1, fc2, out) + ((mixer._modules["in_proj"],) if kind is BaseConv else ()):
            tensors = m._parameters
            if "bias" not in tensors:   # computed, by a parametrization or a pruning
                return None
            own += [tensors.get("weight"), tensors["bias"]]
        if own[0] is None or own[2] is None or own[4] is None or own[0].shape[0] % 16 or own[0].shape[1] % 8:
            return None
        taps = None
        if kind is BaseConv:
            conv = mixer._modules["conv"]
            taps = conv._modules["conv"]._parameters.get("weight")
            if own[6] is None or taps is None or not conv.takes_prompt() or own[6].shape[0] % 16:
                return None
        if own[2].shape[0] != width or own[4].shape[0] != width or own[2].shape[1] % 8 or own[4].shape[1] % 8:
            return None
        w1, b1, w2, b2, wo, bo, wi, bi = own if kind is BaseConv else (*own, None, None)
        return PromptPlan(mixer, norm1, norm2, w1, b1, w2, b2, act, wo, bo, wi, bi, taps, norm1._parameters["weight"], norm2._parameters["weight"])

    def prompt(self, rows, residual, inference_params, plan, next_norm):
        """:meth:`forward` of a prompt with the :meth:`prompt_plan` of this layer: ``rows`` is what ``norm1`` gives (a tensor, or a
        :class:`ops.NormRows`), ``residual`` is updated in place; returns what ``next_norm`` gives, or without one the MLP's output."""
        p: PromptPlan = plan
        x, ss, eps = (rows.x, rows.ss, rows.eps) if type(rows) is ops.NormRows else (rows, None, 0.0)
        B, L, _ = x.shape
        first = (None,) * 7
        if p.taps is not None:
            state = p.mixer.conv._prefill_state(inference_params, B, clear=False)
            if L >= 3 and (state is None or (state.dtype == torch.bfloat16 and state.is_contiguous() and state.data_ptr() % 16 == 0)):
                first = p.in_proj, p.in_bias, p.taps, state, p.out_proj, p.out_bias, p.norm2_weight
        if first[0] is None:
            rows = p.mixer(rows, inference_params=inference_params,
                           finish=lambda x, weight, bias: ops.prompt_add_norm(x, weight, bias, residual, p.norm2_weight, eps=p.norm2.eps))
            x, ss, eps = rows.x, rows.ss, rows.eps
        x, ss = ops.prompt_layer(x, ss, eps, residual, L, *first, p.norm2.eps, p.fc1, p.fc1_bias, p.activation, p.fc2, p.fc2_bias,
                                 None if next_norm is None else next_norm.weight, 0.0 if next_norm is None else next_norm.eps)
        return x if next_norm is None else ops.NormRows(x, ss, next_norm.eps)

    def step(self, hidden_states, residual, inference_params, next_norm):
        """:meth:`forward` for a decode step where :meth:`step_ok`: ``residual`` is updated in place, ``hidden_states`` may be what
        the block before returned, and with ``next_norm`` this one returns what the next block's norm gives.  The norms see the fp32
        stream: the rounding to the activations' dtype comes once, behind the norm's weight."""
        if type(hidden_states) is not ops.NormRows:
            hidden_states, residual = self.norm1(hidden_states, residual=residual, prenorm=True, residual_in_fp32=True, round_input=True)

        def into(norm):
            return lambda x, weight, bias: ops.linear_add_norm(x, weight, bias, residual, norm.weight, eps=norm.eps)

        hidden_states = self.mixer(hidden_states, inference_params=inference_params, finish=into(self.norm2))
        return self.mlp(hidden_states, finish=None if next_norm is None else into(next_norm)), residual

    def forward(self, hidden_states, residual=None, inference_params=None):
        # block.py:134-137: residual = hidden + residual; hidden = norm(residual.to(weight dtype)); residual kept in fp32
        hidden_states, residual = self.norm1(hidden_states, residual=residual, prenorm=True,
                                             residual_in_fp32=self.residual_in_fp32, round_input=True)
        hidden_states = self.mixer(hidden_states, inference_params=inference_params)
        hidden_states, residual = self.norm2(hidden_states, residual=residual, prenorm=True,
                                             residual_in_fp32=self.residual_in_fp32, round_input=True)
        return self.mlp(hidden_states), residual


class _Embeddings(nn.Module):
    def __init__(self, embed_dim, vocab_size, device=None, dtype=None):
        super().__init__()
        self.word_embeddings = nn.Embedding(vocab_size, embed_dim, device=device, dtype=dtype)

    def forward(self, input_ids):
        return self.word_embeddings(input_ids)


class BasedModel(nn.Module):
    def __init__(self, config: BasedConfig, device=None, dtype=None):
        super().__init__()
        self.config = config
        self.embeddings = _Embeddings(config.n_embd, config.padded_vocab_size, device=device, dtype=dtype)
        self.layers = nn.ModuleList([Block(config, i, device=device, dtype=dtype) for i in range(config.n_layer)])
        self.ln_f = RMSNorm(config.n_embd, eps=config.layer_norm_epsilon, device=device, dtype=dtype)

    def allocate_inference_cache(self, batch_size, max_seqlen, dtype=None, **kwargs):
        return {i: layer.allocate_inference_cache(batch_size, max_seqlen, dtype=dtype, **kwargs)
                for i, layer in enumerate(self.layers)}

    def _step_ok(self, h):
        return (h.dim() == 3 and h.shape[1] == 1 and h.shape[0] <= ops.STEP_MAX_ROWS and len(self.layers) > 0
                and ops._decode_rows(h, self.layers[0].mlp.fc1.weight) and not torch.nn.modules.module._has_any_global_hook()
                and all(type(layer) is Block and layer.step_ok(h.shape[-1]) for layer in self.layers))

    def _prompt_plans(self, h):
        """Every layer's plan, or None where a prompt ``h`` has to go through the modules' own forwards."""
        layers = self._modules["layers"]._modules.values()
        if not (h.dim() == 3 and len(layers) > 0 and all(type(layer) is Block for layer in layers) and ops._prompt_rows(h, self.layers[0].mlp.fc1.weight)
                and not torch.nn.modules.module._has_any_global_hook()):
            return None
        plans = [layer.prompt_plan(h.shape[-1]) for layer in layers]
        if any(p is None for p in plans) or not ops.plain_bf16(h, *(w for p in plans for w in p[3:] if torch.is_tensor(w))):
            return None
        return plans

    def forward(self, input_ids, inference_params=None):
        hidden_states, residual = self.embeddings(input_ids), None
        step = inference_params is not None and inference_params.seqlen_offset > 0
        plans = None if step else self._prompt_plans(hidden_states)
        if plans is not None:
            layers, norms = list(self.layers), [p.norm1 for p in plans[1:]] + [None]
            hidden_states, residual = layers[0].norm1(hidden_states, prenorm=True, residual_in_fp32=True, round_input=True)
            for layer, plan, norm in zip(layers, plans, norms):
                hidden_states = layer.prompt(hidden_states, residual, inference_params, plan, norm)
        elif step and self._step_ok(hidden_states):
            following = [layer.norm1 for layer in self.layers[1:]] + [None]
            for layer, norm in zip(self.layers, following):
                hidden_states, residual = layer.step(hidden_states, residual, inference_params, norm)
        else:
            for layer in self.layers:
                hidden_states, residual = layer(hidden_states, residual, inference_params=inference_params)
        # gpt.py:676-690: last add, then the final norm on the sum cast to the weights' dtype
        return self.ln_f(hidden_states, residual=residual, residual_in_fp32=self.config.residual_in_fp32,
                         round_input=True)


class BasedLMHeadModel(GenerationMixin, nn.Module):
    def __init__(self, config: BasedConfig, device=None, dtype=None):
        super().__init__()
        self.config = config
        self.transformer = BasedModel(config, device=device, dtype=dtype)
        self.lm_head = nn.Linear(config.n_embd, config.padded_vocab_size, bias=False, device=device, dtype=dtype)
        self.tie_weights()

    @classmethod
    def from_config(cls, d, device=None, dtype=None):
        return cls(BasedConfig.from_dict(d), device=device, dtype=dtype)

    def load_tensors(self, tensors):
        """Weights by the reference's parameter names (``tensors`` as :class:`based_b200.weights.SafeTensors`)."""
        own = {k: v for k, v in self.state_dict().items() if k != "lm_head.weight"}
        missing = [k for k in own if k not in tensors]
        if missing:
            raise KeyError(f"missing tensors: {missing[:5]}")
        with torch.no_grad():
            for k, v in own.items():
                v.copy_(tensors.get(k, tuple(v.shape)))
        self.tie_weights()

    def tie_weights(self):
        self.lm_head.weight = self.transformer.embeddings.word_embeddings.weight

    def allocate_inference_cache(self, batch_size, max_seqlen, dtype=None, **kwargs):
        return self.transformer.allocate_inference_cache(batch_size, max_seqlen, dtype=dtype, **kwargs)

    def forward(self, input_ids, inference_params=None, num_last_tokens=0):
        """Logits ``[B, L, padded_vocab]`` (the last ``num_last_tokens`` positions when > 0), gpt.py:794-830."""
        hidden_states = self.transformer(input_ids, inference_params=inference_params)
        if num_last_tokens > 0:
            hidden_states = hidden_states[:, -num_last_tokens:]
        return ops.linear(hidden_states, self.lm_head.weight, self.lm_head.bias)
