"""Fused elementwise operations of a LLaMA decoder layer for the token-by-token decode step.

``enable_fused_decode_ops(model)`` swaps pieces of a transformers LLaMA model for single CUDA launches of the C
ABI: RMSNorm (``ade_b200_rmsnorm``), the rotary position embedding of q and k (``ade_b200_rope``), SiLU(gate) * up
(``ade_b200_silu_mul``) and, for single-token steps on a static KV cache, the whole attention step: rotary embedding,
cache write and attention (``ade_b200_attn_decode``).  The arithmetic and the bfloat16 roundings of the first three
are those of the torch operations they replace: rotary embedding and SiLU product give the same bits, RMSNorm adds its
mean of squares in another order, so a last bit can differ; the attention step keeps scores and sums in float32 where
torch's fused attention rounds the probabilities to bfloat16, a difference below the tolerance of the path.  (An
eight-layer 7B model on 4 x 500 tokens is as far from a float64 evaluation, 0.76 % of its logits, with the launches as
without; the two differ by 0.44 %.)  What changes is the number of kernels per token (about sixty per layer fewer),
which at decode sizes is what the time outside the delta application consists of.  Prompts of any length gain as well
(each replaced kernel is a pass over the activations; the same prompts 12.7 -> 9.9 ms), but above ``MAX_ROWS`` token
rows the operations are replaced only where nothing differentiates, traces or listens: gradients of what a layer's
modules return, dispatch modes and tensor subclasses, hooks and wrapped modules all get the original operations.  Other
dtypes, CPU tensors and operands spread over devices take the original code.

The reference has no counterpart: it generates with ``model.generate`` of transformers (src/evaluate.py:241).
"""
from __future__ import annotations

import torch

from . import _lib
from .kernels import _on_device

MAX_ROWS = 512          # token rows (batch * sequence) up to which the fused kernels are used unconditionally
SILU_TYPES = ("SiLU", "SiLUActivation")


def _launch(entry: str, dev: torch.device, *args) -> None:
    """One call of the C entry `entry` on the current stream of `dev`, the device of the tensors (which need not be the current one)."""
    with _on_device(dev):
        _lib.check(getattr(_lib.load(), entry)(*args, torch._C._cuda_getCurrentRawStream(dev.index)), entry)


def _plain_inference(*tensors) -> bool:
    """Nothing records or transforms the operations on these tensors: no gradient, forward-mode or functorch level, no
    tracing, no dispatch mode or tensor subclass (fake tensors, counters) that has to see them.  The reconstructed path of a
    long input is differentiable, so the operations around it have to stay so."""
    if torch.is_grad_enabled() and any(t.requires_grad for t in tensors):
        return False
    if torch._C._len_torch_dispatch_stack() or any(type(t) not in (torch.Tensor, torch.nn.Parameter) for t in tensors):
        return False
    return (torch.autograd.forward_ad._current_level < 0 and torch._C._functorch.peek_interpreter_stack() is None
            and not torch.jit.is_tracing() and not torch.compiler.is_compiling())


def _on_cuda(t: torch.Tensor) -> bool:
    return t.is_cuda


def _rows_ok(t: torch.Tensor, rows: int, *others) -> bool:
    """The kernels take `t` together with `others`: all on one device, and nothing records what is done with them."""
    return (_on_cuda(t) and t.dtype == torch.bfloat16 and rows > 0 and all(o.device == t.device for o in others)
            and (rows <= MAX_ROWS or _plain_inference(t, *others)))


def _passable(mod) -> bool:
    """Nobody would notice that `mod` is not called: no hooks of its own or for all modules, and the forward it came (or was patched) with."""
    m = torch.nn.modules.module
    return not (mod._forward_hooks or mod._forward_pre_hooks or mod._backward_hooks or mod._backward_pre_hooks or m._global_forward_hooks
                or m._global_forward_pre_hooks or m._global_backward_hooks or m._global_backward_pre_hooks
                or mod.__dict__.get("forward") is not mod.__dict__.get("_ade_forward"))


def rmsnorm(x: torch.Tensor, weight: torch.Tensor, eps: float) -> torch.Tensor:
    """LlamaRMSNorm.forward for a bfloat16 CUDA tensor whose last dimension is contiguous."""
    H = x.shape[-1]
    x2 = x.reshape(-1, H)
    if x2.stride(1) != 1:
        x2 = x2.contiguous()
    out = torch.empty((x2.shape[0], H), dtype=torch.bfloat16, device=x.device)
    _launch("ade_b200_rmsnorm", x.device, x2.data_ptr(), weight.data_ptr(), out.data_ptr(), x2.shape[0], H, x2.stride(0), float(eps))
    return out.view(x.shape)


def add_rmsnorm(x: torch.Tensor, residual: torch.Tensor, weight: torch.Tensor, eps: float):
    """(residual + x, LlamaRMSNorm(residual + x)) in one launch: the residual connection of a decoder layer and the
    normalisation that follows it.  Both inputs bfloat16 CUDA with a contiguous last dimension."""
    H = x.shape[-1]
    x2, r2 = x.reshape(-1, H), residual.reshape(-1, H)
    if x2.stride(1) != 1:
        x2 = x2.contiguous()
    if r2.stride(1) != 1:
        r2 = r2.contiguous()
    total = torch.empty((x2.shape[0], H), dtype=torch.bfloat16, device=x.device)
    out = torch.empty_like(total)
    _launch("ade_b200_add_rmsnorm", x.device, x2.data_ptr(), r2.data_ptr(), weight.data_ptr(), total.data_ptr(), out.data_ptr(), x2.shape[0], H,
            x2.stride(0), r2.stride(0), float(eps))
    return total.view(x.shape), out.view(x.shape)


def rope(q: torch.Tensor, k: torch.Tensor, cos: torch.Tensor, sin: torch.Tensor):
    """apply_rotary_pos_emb for q (B, heads, T, hd) and k given as transposed views of (B, T, heads, hd) projections;
    returns contiguous (B, heads, T, hd) tensors."""
    B, hq, T, hd = q.shape
    hk = k.shape[1]
    qo = torch.empty((B, hq, T, hd), dtype=torch.bfloat16, device=q.device)
    ko = torch.empty((B, hk, T, hd), dtype=torch.bfloat16, device=q.device)
    cs_stride = 0 if cos.shape[0] == 1 else T * hd
    # distance between consecutive (batch, token) rows of the projection; a dimension of size 1 reports an arbitrary stride
    rq = q.stride(2) if T > 1 else q.stride(0)
    rk = k.stride(2) if T > 1 else k.stride(0)
    _launch("ade_b200_rope", q.device, q.data_ptr(), k.data_ptr(), cos.data_ptr(), sin.data_ptr(), qo.data_ptr(), ko.data_ptr(), B, T, hq, hk, hd,
            rq, rk, cs_stride)
    return qo, ko


def silu_mul(gate: torch.Tensor, up: torch.Tensor) -> torch.Tensor:
    """act_fn(gate) * up for SiLU, bfloat16, last dimension contiguous (row strides free)."""
    cols = gate.shape[-1]
    g2, u2 = gate.reshape(-1, cols), up.reshape(-1, cols)
    out = torch.empty((g2.shape[0], cols), dtype=torch.bfloat16, device=gate.device)
    _launch("ade_b200_silu_mul", gate.device, g2.data_ptr(), u2.data_ptr(), out.data_ptr(), g2.shape[0], cols, g2.stride(0), u2.stride(0))
    return out.view(*gate.shape[:-1], cols)


def attn_decode(q, k, v, cos, sin, mask, layer, scale: float) -> torch.Tensor:
    """Single-token attention step on a static cache layer: q (B, 1, hq*hd), k / v (B, 1, hk*hd) straight from the
    projections, cos / sin (B or 1, 1, hd), mask None or bool (B, 1, 1, L).  Writes k, v into the layer's cache at its
    running position, advances that position (inside the same launch), returns (B, 1, hq*hd)."""
    B = q.shape[0]
    hk, L, hd = layer.keys.shape[1], layer.keys.shape[2], layer.keys.shape[3]
    hq = q.shape[-1] // hd
    out = torch.empty((B, 1, hq * hd), dtype=torch.bfloat16, device=q.device)
    row = lambda t: t.stride(0) if B > 1 else t.shape[-1]
    ticket = getattr(layer, "_ade_ticket", None)           # counter through which the launch advances the position itself
    if ticket is None or ticket.device != q.device:
        ticket = layer._ade_ticket = torch.zeros(1, dtype=torch.int32, device=q.device)
    _launch("ade_b200_attn_decode", q.device,
            q.data_ptr(), k.data_ptr(), v.data_ptr(), cos.data_ptr(), sin.data_ptr(), None if mask is None else mask.data_ptr(),
            layer.keys.data_ptr(), layer.values.data_ptr(), layer.cumulative_length.data_ptr(), ticket.data_ptr(), out.data_ptr(), B, hq, hk, hd, L,
            row(q), row(k), row(v), 0 if cos.shape[0] == 1 else hd, 0 if mask is None else mask.stride(0), float(scale))
    return out


def _attn_decode_ok(mod, x, cos, mask, layer) -> bool:
    if not (x.is_cuda and x.dtype == torch.bfloat16 and x.dim() == 3 and x.shape[1] == 1 and not mod.training):
        return False
    if type(layer).__name__ != "StaticLayer" or not getattr(layer, "is_initialized", False):
        return False
    kc = layer.keys
    if not (kc.dtype == torch.bfloat16 and kc.is_contiguous() and layer.values.is_contiguous() and kc.shape[0] == x.shape[0]):
        return False
    if any(t.device != x.device for t in (cos, kc, layer.values, layer.cumulative_length)) or (mask is not None and mask.device != x.device):
        return False
    hd = kc.shape[3]
    if hd % 32 or hd > 256 or (7 * hd + kc.shape[2]) * 4 > 48 * 1024 or layer.cumulative_length.dtype != torch.int64:
        return False
    if not (cos.dtype == torch.bfloat16 and cos.dim() == 3 and cos.shape[1:] == (1, hd) and cos.is_contiguous() and cos.shape[0] in (1, x.shape[0])):
        return False
    if mask is not None and not (mask.dtype == torch.bool and mask.dim() == 4 and mask.shape[1] == 1 and mask.shape[2] == 1
                                 and mask.shape[3] == kc.shape[2] and mask.stride(3) == 1 and mask.shape[0] == x.shape[0]):
        return False
    return True


def _rope_layout_ok(x: torch.Tensor) -> bool:
    """(B, heads, T, hd) view of a (B, T, heads, hd) projection: head_dim contiguous, heads hd apart, batch rows T apart."""
    B, h, T, hd = x.shape
    return x.stride(3) == 1 and (h == 1 or x.stride(1) == hd) and (B == 1 or T == 1 or x.stride(0) == T * x.stride(2))


def _rope_ok(q: torch.Tensor, k: torch.Tensor, cos: torch.Tensor, sin: torch.Tensor) -> bool:
    """The launch reads a full table row for every (batch, token): what torch would broadcast is left to it."""
    return (q.dim() == 4 and k.dim() == 4 and _rows_ok(q, q.shape[0] * q.shape[2], k, cos, sin) and k.dtype == torch.bfloat16
            and k.shape[0] == q.shape[0] and k.shape[2:] == q.shape[2:] and q.shape[3] % 2 == 0
            and cos.dtype == sin.dtype == torch.bfloat16 and cos.dim() == 3 and cos.shape == sin.shape and cos.shape[1:] == q.shape[2:]
            and cos.is_contiguous() and sin.is_contiguous() and cos.shape[0] in (1, q.shape[0]) and _rope_layout_ok(q) and _rope_layout_ok(k))


def _norm_ok(x: torch.Tensor, weight: torch.Tensor) -> bool:
    return weight.dtype == torch.bfloat16 and weight.shape == x.shape[-1:] and weight.is_contiguous() and x.stride(-1) == 1


def _add_norm_ok(x: torch.Tensor, residual: torch.Tensor, norm) -> bool:
    """`residual + x` and the LlamaRMSNorm `norm` behind it can be one launch.  Asked about the very tensors that go into it: a
    module in front may have made one of them require a gradient although the layer's input does not."""
    return (_rows_ok(x, x.numel() // x.shape[-1], residual, norm.weight) and residual.dtype == torch.bfloat16 and x.shape == residual.shape
            and _norm_ok(x, norm.weight) and residual.stride(-1) == 1)


def enable_fused_decode_ops(model) -> int:
    """Patch `model` (a transformers LLaMA-architecture causal LM) in place; returns the number of modules patched.
    The rotary embedding is a module-level function of transformers' LLaMA implementation, so that patch is process-wide: LLaMA models
    that were never patched take the launch too, for bfloat16 CUDA inputs with everything on one device (above ``MAX_ROWS`` token rows
    where nothing differentiates or traces); anything else takes the original."""
    from transformers.models.llama import modeling_llama as ml

    if not getattr(ml, "_ade_rope_patched", False):
        original = ml.apply_rotary_pos_emb

        def apply_rotary_pos_emb(q, k, cos, sin, unsqueeze_dim=1):
            if unsqueeze_dim == 1 and _rope_ok(q, k, cos, sin):
                return rope(q, k, cos, sin)
            return original(q, k, cos, sin, unsqueeze_dim)

        ml.apply_rotary_pos_emb = apply_rotary_pos_emb
        ml._ade_rope_patched = True
    n = 0
    for mod in model.modules():
        if isinstance(mod, ml.LlamaAttention) and not hasattr(mod, "_ade_orig_forward"):
            mod._ade_orig_forward = mod.forward

            def attn_forward(hidden_states, position_embeddings=None, attention_mask=None, past_key_values=None, mod=mod, **kw):
                layers = getattr(past_key_values, "layers", None)
                layer = layers[mod.layer_idx] if layers is not None and mod.layer_idx < len(layers) else None
                if (position_embeddings is not None and layer is not None
                        and _attn_decode_ok(mod, hidden_states, position_embeddings[0], attention_mask, layer)):
                    q, k, v = mod.q_proj(hidden_states), mod.k_proj(hidden_states), mod.v_proj(hidden_states)
                    kc, cos, sin = layer.keys, *position_embeddings
                    if (all(t.dtype == torch.bfloat16 and t.stride(-1) == 1 and t.device == hidden_states.device for t in (q, k, v))
                            and q.shape[-1] % kc.shape[3] == 0 and k.shape[-1] == v.shape[-1] == kc.shape[1] * kc.shape[3]
                            and layer.values.shape == kc.shape and sin.shape == cos.shape and sin.dtype == cos.dtype and sin.is_contiguous()
                            and sin.device == hidden_states.device):
                        ctx = attn_decode(q, k, v, cos, sin, attention_mask, layer, mod.scaling)
                        return mod.o_proj(ctx), None
                return mod._ade_orig_forward(hidden_states, position_embeddings=position_embeddings, attention_mask=attention_mask,
                                             past_key_values=past_key_values, **kw)

            mod.forward = attn_forward
            n += 1
        elif isinstance(mod, ml.LlamaRMSNorm) and not hasattr(mod, "_ade_orig_forward"):
            mod._ade_orig_forward = mod.forward

            mod._ade_pre = None                   # (input tensor, its version, its normalisation) left by the layer in front, see below

            def norm_forward(x, mod=mod):
                pre = mod._ade_pre
                if pre is not None:
                    mod._ade_pre = None
                    if x is pre[0] and x._version == pre[1]:
                        return pre[2]
                if _rows_ok(x, x.numel() // x.shape[-1], mod.weight) and _norm_ok(x, mod.weight):
                    return rmsnorm(x, mod.weight, mod.variance_epsilon)
                return mod._ade_orig_forward(x)

            mod.forward = mod._ade_forward = norm_forward
            n += 1
        elif (isinstance(mod, ml.LlamaMLP) and not hasattr(mod, "_ade_orig_forward")
              and type(mod.act_fn).__name__ in SILU_TYPES):
            mod._ade_orig_forward = mod.forward

            def mlp_forward(x, mod=mod):
                if _rows_ok(x, x.numel() // x.shape[-1]):
                    g, u = mod.gate_proj(x), mod.up_proj(x)
                    if (_rows_ok(g, g.numel() // g.shape[-1], u) and u.dtype == torch.bfloat16 and g.shape == u.shape and g.stride(-1) == 1
                            and u.stride(-1) == 1 and type(mod.act_fn).__name__ in SILU_TYPES and _passable(mod.act_fn)):
                        return mod.down_proj(silu_mul(g, u))
                    return mod.down_proj(mod.act_fn(g) * u)
                return mod._ade_orig_forward(x)

            mod.forward = mlp_forward
            n += 1
    # Residual connections: a decoder layer adds the attention output and the MLP output to its input, each time right in
    # front of an RMSNorm (its own post-attention norm; the next layer's input norm, or the model's final norm).  A
    # patched layer does add + norm in one launch each and leaves the second normalisation with the norm module that is
    # about to be asked for it, which recognises the tensor by identity and by its version: a hook or wrapper in between may
    # have edited it in place.
    for lm in model.modules():
        if not isinstance(lm, ml.LlamaModel):
            continue
        layers = list(lm.layers[: lm.config.num_hidden_layers])
        for i, layer in enumerate(layers):
            if hasattr(layer, "_ade_orig_forward") or not isinstance(layer, ml.LlamaDecoderLayer):
                continue
            nxt = layers[i + 1].input_layernorm if i + 1 < len(layers) else lm.norm
            if not all(hasattr(nm, "_ade_pre") for nm in (layer.input_layernorm, layer.post_attention_layernorm, nxt)):
                continue
            layer._ade_orig_forward = layer.forward

            def layer_forward(hidden_states, attention_mask=None, position_ids=None, past_key_values=None, use_cache=False,
                              position_embeddings=None, layer=layer, nxt=nxt, **kw):
                post = layer.post_attention_layernorm
                if not (_rows_ok(hidden_states, hidden_states.numel() // hidden_states.shape[-1]) and not layer.training):
                    return layer._ade_orig_forward(hidden_states, attention_mask=attention_mask, position_ids=position_ids,
                                                   past_key_values=past_key_values, use_cache=use_cache,
                                                   position_embeddings=position_embeddings, **kw)
                h = layer.input_layernorm(hidden_states)
                a, _ = layer.self_attn(hidden_states=h, attention_mask=attention_mask, position_ids=position_ids,
                                       past_key_values=past_key_values, use_cache=use_cache, position_embeddings=position_embeddings, **kw)
                if _add_norm_ok(a, hidden_states, post) and hasattr(post, "_ade_pre") and _passable(post):
                    s1, h2 = add_rmsnorm(a, hidden_states, post.weight, post.variance_epsilon)
                else:
                    s1 = hidden_states + a
                    h2 = post(s1)
                m = layer.mlp(h2)
                if torch.is_inference_mode_enabled() or not _add_norm_ok(m, s1, nxt):     # inference tensors do not count their versions
                    return s1 + m
                s2, h3 = add_rmsnorm(m, s1, nxt.weight, nxt.variance_epsilon)
                nxt._ade_pre = (s2, s2._version, h3)
                return s2

            layer.forward = layer_forward
            n += 1
    return n
