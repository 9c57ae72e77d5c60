"""Llama decoder re-hosted on CUDA tensors around the B200 KV-cache path.

The caller of the hot path, kept in the reference's shape (pace/llm/models/llama.py): per layer
q/k/v projection -> RoPE -> ``kv_cache.update_cache`` -> ``MultiHeadAttention`` -> o_proj
(llama.py:111-170), model forward slicing off what is already cached (llama.py:270-318).
Parameter names match the reference's state dict, so its weights load unchanged.

Differences that come from the path being on the GPU:
  * no ``repeat_kv``: the cache holds the KV heads, the attention kernels are GQA-native;
  * no 4-D additive mask: causality and left padding reach the kernels as per-sequence integers
    (``kv_start`` = padded positions, the causal tail follows from the cached lengths);
  * RoPE is fused into the append kernel (``update_cache_rope``); a residual sum and the norm behind it are one
    kernel, the activation of the MLP another; projections are library products, one for weights that lie side
    by side (query, key and value; gate and up).  Where gradients, hooks or replaced modules are in play the
    modules are called one by one;
  * ``forward_tokens`` takes only the NEW tokens and allows ragged counts per sequence, which
    batched speculative decoding needs; ``forward`` is the reference signature on top of it.
"""
from types import SimpleNamespace
from typing import Dict, Optional, Sequence

import numpy as np
import torch
import torch.nn.functional as F
from torch import nn
from torch.autograd import forward_ad
from torch.nn.modules.module import _has_any_global_hook

from pace_b200 import _C
from pace_b200.llm.cache import KVCacheBase, KVCacheManager
from pace_b200.llm.outputs import ModelOutput
from pace_b200.llm.registry import model_registry
from pace_b200.ops import MultiHeadAttention, RotaryEmbedding
from pace_b200.ops.linear import linear


def _untouched(m: nn.Module, cls: type) -> bool:
    """Whether calling m is nothing but ``cls.forward``: no other class, no forward of its own, no hooks."""
    return type(m) is cls and "forward" not in m.__dict__ and not (
        m._forward_hooks or m._forward_pre_hooks or m._backward_hooks or m._backward_pre_hooks or _has_any_global_hook())


def _no_graph(*tensors: torch.Tensor) -> bool:
    """Whether kernels that autograd, transforms and tracers do not see may run over these tensors."""
    if forward_ad._current_level >= 0 or torch._C._are_functorch_transforms_active() or torch.jit.is_tracing() or torch.compiler.is_compiling():
        return False
    grad = torch.is_grad_enabled()
    return all(type(t) in (torch.Tensor, nn.Parameter) and t.is_cuda and t.dtype == torch.bfloat16 and t.numel() > 0 and
               not (grad and t.requires_grad) for t in tensors)


def _fusable(x: torch.Tensor, *modules: nn.Module) -> bool:
    """The same for plain linears over x that nobody has replaced or hooked."""
    return all(_untouched(m, nn.Linear) and m.bias is None for m in modules) and _no_graph(x, *(m.weight for m in modules))


def _side_by_side(*modules: nn.Module) -> Optional[torch.Tensor]:
    """The weights of linears over the same input as one matrix, where they lie behind one another in memory (``_lay_out``)."""
    w = [m.weight for m in modules]
    at, store = w[0].data_ptr(), w[0].untyped_storage()
    for x in w:
        if x.data_ptr() != at or not x.is_contiguous() or x.shape[1] != w[0].shape[1] or x.dtype != w[0].dtype or \
                x.untyped_storage().data_ptr() != store.data_ptr():
            return None
        at += x.numel() * x.element_size()
    return w[0].as_strided((sum(x.shape[0] for x in w), w[0].shape[1]), (w[0].shape[1], 1))


def _lay_out(*modules: nn.Module) -> None:
    """Puts the weights of linears over the same input behind one another, so that a step makes one product of them."""
    if any(type(m) is not nn.Linear or type(m.weight) is not nn.Parameter or not m.weight.is_cuda or m.weight.dtype != torch.bfloat16 or
           m.weight.is_inference() != torch.is_inference_mode_enabled() for m in modules):
        return
    w = [m.weight for m in modules]
    if any(x.shape[1] != w[0].shape[1] or x.device != w[0].device for x in w) or _side_by_side(*modules) is not None:
        return
    both, at = torch.cat([x.data for x in w]), 0
    for x in w:
        x.data = both[at: at + x.shape[0]]
        at += x.shape[0]


def _rows(x: torch.Tensor, dtype: torch.dtype) -> torch.Tensor:
    """x as the append reads it: that type, heads of consecutive elements, rows at 16 bytes (what a replaced projection leaves may differ)."""
    if x.dtype != dtype or x.stride(-1) != 1 or any(s % 8 for s in x.stride()[:-1]) or x.data_ptr() % 16:
        x = x.to(dtype).clone(memory_format=torch.contiguous_format)
    return x


def _add_norm(x: torch.Tensor, y: Optional[torch.Tensor], norm: "RMSNorm"):
    """(x + y, its norm); without y (x, its norm)."""
    W = x.shape[-1]
    if _untouched(norm, RMSNorm) and _no_graph(x, norm.weight, x if y is None else y) and W % 8 == 0 and W <= 8192 and \
            norm.weight.is_contiguous() and x.is_contiguous() and (y is None or (y.is_contiguous() and y.shape == x.shape)) and \
            not any(t.data_ptr() % 16 for t in ((x, norm.weight) if y is None else (x, y, norm.weight))):
        s, out = x if y is None else torch.empty_like(x), torch.empty_like(x)
        torch.ops.pace_b200.add_norm(x, y, norm.weight, None if y is None else s, out, norm.eps)
        return s, out
    s = x if y is None else x + y
    return s, norm(s)


class _FusedLinear(nn.Module):
    """Holds ``linear.weight`` like the reference's fused linear + activation operators."""

    def __init__(self, in_features: int, out_features: int):
        super().__init__()
        self.linear = nn.Linear(in_features, out_features, bias=False)


class RMSNorm(nn.Module):
    def __init__(self, hidden: int, eps: float):
        super().__init__()
        self.weight = nn.Parameter(torch.ones(hidden))
        self.eps = eps

    def forward(self, x):
        return F.rms_norm(x, (x.shape[-1],), self.weight, self.eps)


class LlamaMLP(nn.Module):
    """down(up(x) * silu(gate(x))) (reference MergedMLP with gate, pace/ops/mlp.py:73-79)."""

    def __init__(self, hidden: int, inter: int):
        super().__init__()
        self.up_proj = _FusedLinear(hidden, inter)
        self.gate_proj = _FusedLinear(hidden, inter)
        self.down_proj = nn.Linear(inter, hidden, bias=False)

    def forward(self, x):
        gate, up = self.gate_proj.linear, self.up_proj.linear
        if _fusable(x, gate, up):
            w, n = _side_by_side(gate, up), gate.weight.shape[0]
            if w is not None and up.weight.shape[0] == n and n % 8 == 0:
                both = linear(x, w).view(-1, 2 * n)
                act = torch.empty(both.shape[0], n, dtype=x.dtype, device=x.device)
                torch.ops.pace_b200.glu(both, act, _C.ACT_SILU)
                return self.down_proj(act.view(*x.shape[:-1], n))
        return self.down_proj(up(x) * F.silu(gate(x)))


class FusedRope:
    """What a decoder layer needs to rotate and append in one kernel: the operator (tables) and the
    table row of every new token."""

    def __init__(self, op: RotaryEmbedding, table_row: torch.Tensor):
        self.op, self.table_row = op, table_row


FUSED_ROPE = True     # RoPE fused into the append kernel; False keeps it as separate elementwise ops (tests compare the two)


class LlamaAttention(nn.Module):
    def __init__(self, config):
        super().__init__()
        self.hidden_size = config.hidden_size
        self.num_heads = config.num_attention_heads
        self.head_dim = self.hidden_size // self.num_heads
        self.num_key_value_heads = config.num_key_value_heads
        self.q_proj = nn.Linear(self.hidden_size, self.num_heads * self.head_dim, bias=False)
        self.k_proj = nn.Linear(self.hidden_size, self.num_key_value_heads * self.head_dim, bias=False)
        self.v_proj = nn.Linear(self.hidden_size, self.num_key_value_heads * self.head_dim, bias=False)
        self.o_proj = nn.Linear(self.hidden_size, self.hidden_size, bias=False)
        self.attention = MultiHeadAttention()

    def project(self, hidden: torch.Tensor):
        """Query, key and value heads ``[..., heads, D]``; one product where the weights lie side by side, otherwise the modules' own."""
        parts = (self.q_proj, self.k_proj, self.v_proj)
        w = _side_by_side(*parts) if _fusable(hidden, *parts) else None
        x = linear(hidden, w).split([m.weight.shape[0] for m in parts], -1) if w is not None else [m(hidden) for m in parts]
        return [t.unflatten(-1, (-1, self.head_dim)) for t in x]

    def forward(self, hidden_states, position_embeddings, kv_cache: KVCacheBase, kv_start=None, n_new=None,
                q_lens=None):
        bsz, q_len, _ = hidden_states.size()
        q, k, v = self.project(hidden_states)
        # the hot path: rotate, append, then attend over the cache (llama.py:146-165)
        if isinstance(position_embeddings, FusedRope):
            q, key_h, value_h = kv_cache.update_cache_rope(q, k, v, position_embeddings.table_row,
                                                           position_embeddings.op, n_new_per_seq=n_new)
        else:
            q, k = position_embeddings(query=q.transpose(1, 2), key=k.transpose(1, 2))
            key_h, value_h = kv_cache.update_cache(k, v.transpose(1, 2), concat_dim=2, n_new_per_seq=n_new)
        out = self.attention(q, key_h, value_h, attention_mask=None, kv_start=kv_start, q_lens=q_lens)
        out = out.transpose(1, 2).reshape(bsz, q_len, -1)
        return self.o_proj(out)

    def forward_packed(self, hidden: torch.Tensor, pk: "Packed", kv_cache: KVCacheBase) -> torch.Tensor:
        """``hidden`` [T, hidden]: the step's tokens of all sequences, back to back."""
        q, k, v = (_rows(t, pk.q.dtype) for t in self.project(hidden))
        q, key_h, value_h = kv_cache.update_cache_rope_packed(q, k, v, pk.row_at, pk.counts, pk.q_lens, pk.rope.table_row, pk.rope.op, pk.q)
        out = self.attention(q, key_h, value_h, attention_mask=None, q_lens=pk.q_lens)
        return self.o_proj(out.transpose(1, 2).reshape(-1, self.num_heads * self.head_dim).index_select(0, pk.staged))


class Packed:
    """One scheduler step's tokens without padding: sequence b's new tokens are rows ``row_at[b]`` .. of the flat
    list, which the projections, norms and the MLP run on.  The append kernel takes keys and values from there
    and puts the rotated queries into ``q`` [B, n_max, heads, D], shared by all layers (the attention kernels
    address a sequence's rows by a batch stride); ``staged[i]`` is token i's row of that form.  What the
    device needs of all this travels in one copy that nothing waits for."""

    def __init__(self, counts: Sequence[int], cached: Sequence[int], rope: RotaryEmbedding, cfg, device,
                 max_positions: int, tokens: Optional[torch.Tensor] = None):
        self.counts = [int(c) for c in counts]
        B, n_max = len(self.counts), max(self.counts)
        self.n_max = n_max
        n = np.asarray(self.counts, dtype=np.int64)
        cu = np.concatenate([[0], np.cumsum(n)])
        T = int(cu[-1])
        bidx = np.repeat(np.arange(B), n)
        self.live = [b for b, c in enumerate(self.counts) if c]
        parts = [np.asarray(list(cached), dtype=np.int64), cu[1:][n > 0] - 1, np.asarray(self.live, dtype=np.int64),
                 bidx * n_max + np.arange(T) - cu[:-1][bidx], np.concatenate([n, cu[:-1]]).astype(np.int32).view(np.int64)]
        if tokens is not None and tokens.device.type == "cpu" and tokens.dim() == 1 and tokens.dtype in (torch.int32, torch.int64):
            parts.append(tokens.numpy().astype(np.int64))
        host = torch.from_numpy(np.concatenate(parts))
        dev = host.pin_memory().to(device, non_blocking=True) if torch.device(device).type == "cuda" else host.to(device)
        views = dev.split([len(p) for p in parts])
        base, self.last_rows, self.live_rows, self.staged = views[:4]      # last_rows: every live sequence's last token
        self.q_lens, self.row_at = views[4].view(torch.int32).split(B)
        self.tokens = views[5] if len(views) > 5 else tokens
        pos = (base.unsqueeze(1) + torch.arange(n_max, device=device).unsqueeze(0)).clamp_(max=max_positions - 1)
        self.rope = FusedRope(rope, rope.table_rows(pos))
        self.q = torch.zeros(B, n_max, cfg.num_attention_heads, cfg.hidden_size // cfg.num_attention_heads, dtype=torch.bfloat16, device=device)


class LlamaDecoderLayer(nn.Module):
    def __init__(self, config):
        super().__init__()
        self.input_layernorm = RMSNorm(config.hidden_size, config.rms_norm_eps)
        self.self_attn = LlamaAttention(config)
        self.mlp = LlamaMLP(config.hidden_size, config.intermediate_size)
        self.post_attention_layernorm = RMSNorm(config.hidden_size, config.rms_norm_eps)

    def forward(self, hidden_states, position_embeddings, kv_cache, kv_start=None, n_new=None, q_lens=None):
        h, y = self.parts(hidden_states, None, lambda n: self.self_attn(n, position_embeddings, kv_cache, kv_start, n_new, q_lens))
        return h + y

    def forward_packed(self, hidden, pk, kv_cache):
        h, y = self.parts(hidden, None, lambda n: self.self_attn.forward_packed(n, pk, kv_cache))
        return h + y

    def parts(self, x, y, attend):
        """The layer over x + y (y may be None) as two summands, whose sum the next norm takes up."""
        h, n = _add_norm(x, y, self.input_layernorm)
        h, n = _add_norm(h, attend(n), self.post_attention_layernorm)
        return h, self.mlp(n)

    @property
    def plain(self) -> bool:
        return _untouched(self, LlamaDecoderLayer)


class LlamaModel(nn.Module):
    def __init__(self, config):
        super().__init__()
        self.embed_tokens = nn.Embedding(config.vocab_size, config.hidden_size, getattr(config, "pad_token_id", None))
        self.layers = nn.ModuleList([LlamaDecoderLayer(config) for _ in range(config.num_hidden_layers)])
        self.rotary_emb = RotaryEmbedding(getattr(config, "rope_scaling", None),
                                          config.hidden_size // config.num_attention_heads,
                                          config.max_position_embeddings, config.rope_theta)
        self.norm = RMSNorm(config.hidden_size, config.rms_norm_eps)

    def forward_tokens(self, new_ids: torch.Tensor, kv_cache: KVCacheManager, position_ids: torch.Tensor,
                       kv_start: Optional[torch.Tensor] = None, n_new: Optional[Sequence[int]] = None):
        hidden = self.embed_tokens(new_ids)
        if FUSED_ROPE and hidden.dtype == torch.bfloat16:
            rope = FusedRope(self.rotary_emb, self.rotary_emb.table_rows(position_ids))
        else:
            rope = self.rotary_emb(hidden, position_ids)
        q_lens = None
        if isinstance(n_new, torch.Tensor):
            q_lens = n_new           # device-resident counts: used as they are, by the append and by the attention
        elif n_new is not None:
            q_lens = torch.tensor(list(n_new), dtype=torch.int32, device=new_ids.device)
        y = None
        for idx, layer in enumerate(self.layers):
            if getattr(layer, "plain", False):
                hidden, y = layer.parts(hidden, y, lambda n: layer.self_attn(n, rope, kv_cache[idx], kv_start, n_new, q_lens))
            else:
                hidden, y = layer(hidden if y is None else hidden + y, rope, kv_cache[idx], kv_start, n_new, q_lens), None
        kv_cache.commit()        # deferred decode appends: one launch advances every layer (a no-op otherwise)
        return _add_norm(hidden, y, self.norm)[1]

    def forward_packed(self, tokens: torch.Tensor, pk: "Packed", kv_cache: KVCacheManager) -> torch.Tensor:
        hidden = self.embed_tokens(tokens)
        y = None
        for idx, layer in enumerate(self.layers):
            if type(layer) is LlamaDecoderLayer and "forward_packed" not in layer.__dict__:
                hidden, y = layer.parts(hidden, y, lambda n: layer.self_attn.forward_packed(n, pk, kv_cache[idx]))
            else:
                hidden, y = layer.forward_packed(hidden if y is None else hidden + y, pk, kv_cache[idx]), None
        kv_cache.commit()
        return _add_norm(hidden, y, self.norm)[1]


class LlamaForCausalLM(nn.Module):
    def __init__(self, config):
        super().__init__()
        self.config = config
        self.model = LlamaModel(config)
        self.vocab_size = config.vocab_size
        self.lm_head = nn.Linear(config.hidden_size, config.vocab_size, bias=False)

    # -- the reference signature (llama.py:428-440) -----------------------------------------
    def forward(self, input_ids: torch.LongTensor, kv_cache: KVCacheManager, attention_mask: torch.Tensor,
                inputs_embeds=None) -> ModelOutput:
        """``input_ids`` is the whole history; what the cache already holds is sliced off
        (llama.py:284-286).  ``attention_mask`` is the 2-D 0/1 mask; zeros on the left are padding."""
        if inputs_embeds is not None:
            raise NotImplementedError("inputs_embeds is not supported")
        past = len(kv_cache)
        new_ids = input_ids[:, past:]
        mask = attention_mask.to(input_ids.device)
        position_ids = mask.long().cumsum(-1) - 1
        position_ids.masked_fill_(mask == 0, 1)
        position_ids = position_ids[:, past: past + new_ids.shape[1]]
        kv_start = None
        if bool((mask == 0).any()):
            kv_start = (mask.cumsum(-1) == 0).sum(-1).to(torch.int32)
        hidden = self.model.forward_tokens(new_ids, kv_cache, position_ids, kv_start)
        return ModelOutput(logits=self.lm_head(hidden))

    # -- ragged form used by batched speculative decoding ---------------------------------------
    def forward_ragged(self, new_ids: torch.Tensor, n_new: Sequence[int], kv_cache: KVCacheManager) -> ModelOutput:
        """``new_ids`` [B, n_max] holds, left-aligned, ``n_new[b]`` new tokens of sequence b; positions
        continue from each sequence's cached length."""
        cached = kv_cache[0].seq_lens if kv_cache[0].seq_lens else [0] * new_ids.shape[0]
        base = torch.tensor(cached, dtype=torch.long, device=new_ids.device).unsqueeze(1)
        position_ids = base + torch.arange(new_ids.shape[1], device=new_ids.device).unsqueeze(0)
        position_ids.clamp_(max=self.config.max_position_embeddings - 1)
        ragged = None if all(n == new_ids.shape[1] for n in n_new) else list(n_new)
        hidden = self.model.forward_tokens(new_ids, kv_cache, position_ids, None, ragged)
        return ModelOutput(logits=self.lm_head(hidden))


    def forward_device_ragged(self, new_ids: torch.Tensor, n_new: torch.Tensor, kv_cache: KVCacheManager,
                              slots: Optional[torch.Tensor] = None) -> ModelOutput:
        """``forward_ragged`` with the counts on the device: ``n_new`` is a CUDA int32 ``[B]`` tensor (the
        output of a kernel), positions continue from the lengths the device holds, and nothing is read
        back - the host never learns how many tokens each sequence took.  The cache must exist already
        (a prompt pass has run)."""
        pool = kv_cache.pool
        base = pool.seq_len()[0].index_select(0, kv_cache.slots_dev.long()).long().unsqueeze(1)
        position_ids = base + torch.arange(new_ids.shape[1], device=new_ids.device).unsqueeze(0)
        position_ids.clamp_(max=self.config.max_position_embeddings - 1)
        hidden = self.model.forward_tokens(new_ids, kv_cache, position_ids, None, n_new)
        return ModelOutput(logits=self.lm_head(hidden))

    # -- packed form used by continuous batching ----------------------------------------------------
    def forward_packed(self, tokens: torch.Tensor, counts: Sequence[int], kv_cache: KVCacheManager,
                       rows: Optional[Sequence[int]] = None) -> ModelOutput:
        """``tokens`` [T] holds the new tokens of every sequence back to back, ``counts[b]`` of them for
        sequence b (zero for a sequence that sits this step out); positions continue from each
        sequence's cached length.  Returns the logits of the LAST new token of every sequence that had
        any, as ``[B, vocab]`` (rows of idle sequences are zero): the LM head runs on those rows only.
        With ``rows`` (places in ``tokens``) it returns the logits of those instead, ``[len(rows), vocab]``."""
        B = len(counts)
        device = self.lm_head.weight.device
        cached = kv_cache[0].seq_lens if kv_cache[0].seq_lens else [0] * B
        pk = Packed(counts, cached, self.model.rotary_emb, self.config, device, self.config.max_position_embeddings, tokens)
        hidden = self.model.forward_packed(pk.tokens.to(device), pk, kv_cache)
        if rows is not None:
            return ModelOutput(logits=self.lm_head(hidden[torch.tensor(list(rows), dtype=torch.long, device=hidden.device)]))
        last = self.lm_head(hidden.index_select(0, pk.last_rows))
        if len(pk.live) == B:
            return ModelOutput(logits=last)
        logits = torch.zeros(B, self.vocab_size, dtype=last.dtype, device=hidden.device)
        return ModelOutput(logits=logits.index_copy_(0, pk.live_rows, last))

    def _apply(self, fn, recurse=True):
        out = super()._apply(fn, recurse)
        self._lay_out()
        return out

    def _lay_out(self) -> None:
        """Weights that a step multiplies the same rows by lie side by side: query, key and value; gate and up."""
        for layer in self.model.layers:
            if type(layer) is LlamaDecoderLayer and type(layer.self_attn) is LlamaAttention:
                _lay_out(layer.self_attn.q_proj, layer.self_attn.k_proj, layer.self_attn.v_proj)
            if type(layer) is LlamaDecoderLayer and type(layer.mlp) is LlamaMLP and \
                    type(layer.mlp.gate_proj) is type(layer.mlp.up_proj) is _FusedLinear:
                _lay_out(layer.mlp.gate_proj.linear, layer.mlp.up_proj.linear)

    def load_weights(self, tensors: Dict[str, torch.Tensor]) -> None:
        """Checkpoint names: the reference's state dict, or the plain ``mlp.up_proj.weight`` form of it."""
        fused = {f"{n}.weight": f"{n}.linear.weight" for n, m in self.named_modules() if isinstance(m, _FusedLinear)}
        renamed = {fused.get(k, k): v for k, v in tensors.items() if not k.endswith("rotary_emb.inv_freq")}
        if "lm_head.weight" not in renamed and "model.embed_tokens.weight" in renamed:
            renamed["lm_head.weight"] = renamed["model.embed_tokens.weight"]     # tied embeddings
        self.load_state_dict(renamed, strict=True)
        self._lay_out()


def _from_config_json(config: dict, dtype: torch.dtype) -> LlamaForCausalLM:
    cfg = SimpleNamespace(**config)
    cfg.num_key_value_heads = getattr(cfg, "num_key_value_heads", None) or cfg.num_attention_heads
    cfg.rope_theta = getattr(cfg, "rope_theta", 10000.0)
    cfg.pad_token_id = getattr(cfg, "pad_token_id", None)
    return LlamaForCausalLM(cfg).to(dtype)


model_registry.register("LlamaForCausalLM", _from_config_json)


def random_init_(model: nn.Module, seed: int, std: float = 0.02) -> nn.Module:
    """N(0, std) weights from a seed (norm weights stay at one): the BASELINE configs' synthetic models."""
    g = torch.Generator(device="cpu").manual_seed(seed)
    with torch.no_grad():
        for p in model.parameters():
            if p.dim() >= 2:
                p.copy_((torch.randn(p.shape, generator=g) * std).to(p.dtype))
    return model
