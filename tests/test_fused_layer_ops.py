"""The patched decoder layer (`decode_ops.enable_fused_decode_ops`) against the unpatched one where something looks at, edits or
differentiates through what lies between its modules.  600 token rows: above the limit up to which the kernels are unconditional.

Every case runs on the GPU and, with torch stand-ins for the four launches (fresh tensors outside autograd, as a launch through raw
pointers leaves them), on the CPU: what is tested is when a launch may take the place of the operations, not its arithmetic."""
from __future__ import annotations

import copy

import pytest
import torch

from ade_b200 import decode_ops


def _norm(x, weight, eps):
    x32 = x.float()
    return weight * (x32 * torch.rsqrt(x32.pow(2).mean(-1, keepdim=True) + eps)).to(x.dtype)


def _rot(t):
    return torch.cat((-t[..., t.shape[-1] // 2:], t[..., :t.shape[-1] // 2]), -1)


STAND_INS = {
    "rmsnorm": _norm,
    "add_rmsnorm": lambda x, res, weight, eps: (res + x, _norm(res + x, weight, eps)),
    "rope": lambda q, k, cos, sin: tuple(t * cos.unsqueeze(1) + _rot(t) * sin.unsqueeze(1) for t in (q, k)),
    "silu_mul": lambda g, u: torch.nn.functional.silu(g) * u,
}


@pytest.fixture(params=["cpu", pytest.param("cuda", marks=pytest.mark.gpu)])
def dev(request, monkeypatch):
    """(device of the case, names of the launches or stand-ins that were taken)."""
    launches = []
    for name, stand_in in STAND_INS.items():
        fn = torch.no_grad()(stand_in) if request.param == "cpu" else getattr(decode_ops, name)
        monkeypatch.setattr(decode_ops, name, lambda *a, fn=fn, name=name: launches.append(name) or fn(*a))
    if request.param == "cpu":
        monkeypatch.setattr(decode_ops, "_on_cuda", lambda t: True)
    return request.param, launches


def _models(dev, seed=0):
    """(patched, unpatched) frozen copies of one small LLaMA model in eval mode."""
    from transformers import LlamaConfig, LlamaForCausalLM

    cfg = LlamaConfig(hidden_size=256, intermediate_size=512, num_hidden_layers=2, num_attention_heads=4, num_key_value_heads=4, vocab_size=512,
                      max_position_embeddings=1024)
    torch.manual_seed(seed)
    plain = LlamaForCausalLM(cfg).to(torch.bfloat16).eval().to(dev)
    plain.requires_grad_(False)
    patched = copy.deepcopy(plain)
    decode_ops.enable_fused_decode_ops(patched)
    return patched, plain


def _ids(dev, seed=1):
    return torch.randint(0, 512, (2, 300), generator=torch.Generator().manual_seed(seed)).to(dev)


def _rel(a, b):
    return float((a.float() - b.float()).norm() / b.float().norm())


@pytest.mark.parametrize("name", ["self_attn.o_proj", "self_attn.q_proj", "mlp.up_proj", "mlp.gate_proj", "mlp.down_proj"])
def test_gradient_of_one_trainable_module(dev, name):
    """One trainable weight inside a layer: the layer's input requires no gradient, what its modules return does.  A unit in the last
    place of bf16 is 2^-8 of a value and two layers of roundings lie between the weight and the result: 5 per cent."""
    dev, _ = dev
    grads = []
    for model in _models(dev):
        w = model.model.layers[0].get_submodule(name).weight
        w.requires_grad_(True)
        model(input_ids=_ids(dev), use_cache=False).logits.float().square().mean().backward()
        grads.append(w.grad)
    got, want = grads
    assert got is not None and float(want.float().norm()) > 0 and _rel(got, want) < 5e-2


def test_fused_where_nothing_differentiates(dev):
    """The launches are taken on long inputs of a frozen model, with gradients enabled too."""
    dev, launches = dev
    patched, plain = _models(dev)
    with torch.no_grad():
        want = plain(input_ids=_ids(dev), use_cache=False).logits
    launches.clear()
    got = patched(input_ids=_ids(dev), use_cache=False).logits
    assert launches.count("add_rmsnorm") == 4 and launches.count("silu_mul") == 2 and launches.count("rope") == 2
    assert _rel(got, want) < 2e-2


def test_operands_on_another_device_are_left_to_torch(monkeypatch):
    """A model spread over devices: a norm weight, a residual, cos / sin or a cache elsewhere cannot be passed to a launch as a pointer."""
    monkeypatch.setattr(decode_ops, "_on_cuda", lambda t: True)
    x = torch.zeros(2, 4, 8, dtype=torch.bfloat16)
    away = torch.zeros(2, 4, 8, dtype=torch.bfloat16, device="meta")
    norm = torch.nn.Module()
    for weight, residual, ok in ((x[0, 0], x, True), (away[0, 0], x, False), (x[0, 0], away, False)):
        norm.weight = torch.nn.Parameter(weight, requires_grad=False)
        assert decode_ops._add_norm_ok(x, residual, norm) is ok
    assert decode_ops._rows_ok(x, 8, x, x) and not decode_ops._rows_ok(x, 8, x, away)

    class Layer:
        is_initialized = True
        keys = values = torch.zeros(2, 1, 16, 32, dtype=torch.bfloat16)
        cumulative_length = torch.zeros(1, dtype=torch.int64)

    Layer.__name__ = "StaticLayer"
    monkeypatch.setattr(torch.Tensor, "is_cuda", property(lambda t: True))
    step, cos, mod = torch.zeros(2, 1, 32, dtype=torch.bfloat16), torch.zeros(1, 1, 32, dtype=torch.bfloat16), torch.nn.Module().eval()
    assert decode_ops._attn_decode_ok(mod, step, cos, None, Layer())
    assert not decode_ops._attn_decode_ok(mod, step, cos.to("meta"), None, Layer())


def test_launches_go_to_the_device_of_the_tensors(monkeypatch):
    """Every launch is made with the tensors' device current and on that device's current stream."""
    import contextlib
    import types

    current, seen = [], []

    @contextlib.contextmanager
    def on_device(d):
        current.append(d)
        yield
        current.pop()

    class Lib:
        def __getattr__(self, entry):
            return lambda *a: seen.append((entry, list(current), a[-1])) or 0

    monkeypatch.setattr(decode_ops, "_on_device", on_device)
    monkeypatch.setattr(decode_ops._lib, "load", Lib)
    monkeypatch.setattr(torch._C, "_cuda_getCurrentRawStream", lambda index: ("stream of", index), raising=False)
    x = torch.zeros(2, 4, 8, dtype=torch.bfloat16)
    cache = types.SimpleNamespace(keys=torch.zeros(2, 1, 16, 8), values=torch.zeros(2, 1, 16, 8), cumulative_length=torch.zeros(1, dtype=torch.int64))
    decode_ops.rmsnorm(x, x[0, 0], 1e-6)
    decode_ops.add_rmsnorm(x, x, x[0, 0], 1e-6)
    decode_ops.silu_mul(x, x)
    decode_ops.rope(x.unsqueeze(1), x.unsqueeze(1), x[:1], x[:1])
    decode_ops.attn_decode(x[:, :1], x[:, :1], x[:, :1], x[:1, :1], x[:1, :1], None, cache, 1.0)
    assert [s[0] for s in seen] == [f"ade_b200_{n}" for n in ("rmsnorm", "add_rmsnorm", "silu_mul", "rope", "attn_decode")]
    assert all(s[1] == [x.device] and s[2] == ("stream of", x.device.index) for s in seen)


@pytest.mark.parametrize("name", ["post_attention_layernorm", "mlp.act_fn", "input_layernorm", "mlp"])
@pytest.mark.parametrize("how", ["hook", "pre_hook", "global", "wrapped"])
def test_modules_somebody_listens_to_are_called(dev, name, how):
    """Hooks on a module of the layer, hooks for all modules, and a forward that was wrapped: they see as many calls as in the
    unpatched model, and what a hook puts in place of an output arrives."""
    dev, _ = dev
    counts, logits = [], []
    for model in _models(dev):
        mod, seen, handle = model.model.layers[0].get_submodule(name), [], None
        if how == "hook":
            mod.register_forward_hook(lambda m, a, out: seen.append(1) or out * 1.5)
        elif how == "pre_hook":
            mod.register_forward_pre_hook(lambda m, a: seen.append(1))
        elif how == "global":
            handle = torch.nn.modules.module.register_module_forward_hook(lambda m, a, out: seen.append(1) if m is mod else None)
        else:
            inner = mod.forward
            mod.forward = lambda *a, **k: seen.append(1) or inner(*a, **k)
        try:
            with torch.no_grad():
                logits.append(model(input_ids=_ids(dev), use_cache=False).logits)
        finally:
            if handle is not None:
                handle.remove()
        counts.append(len(seen))
    assert counts[0] == counts[1] == 1
    assert _rel(*logits) < 2e-2


@pytest.mark.parametrize("mode", [torch.no_grad, torch.inference_mode])
@pytest.mark.parametrize("rows", [(2, 300), (1, 20)])
def test_hidden_state_edited_in_place_between_layers(dev, mode, rows):
    """A forward hook that adds to a layer's output in place (steering vectors, features added at some layers) leaves the tensor's identity
    as it is; the norm behind it normalises the edited values."""
    dev, _ = dev
    logits, g = [], torch.Generator().manual_seed(3)
    ids, steer = torch.randint(0, 512, rows, generator=g).to(dev), torch.randn(256, generator=g).to(torch.bfloat16).to(dev)
    for model in _models(dev):
        model.model.layers[0].register_forward_hook(lambda m, a, out: (out.add_(steer), None)[1])
        with mode():
            logits.append(model(input_ids=ids, use_cache=False).logits.clone())
    assert _rel(*logits) < 2e-2


def test_dispatch_modes_and_tensor_subclasses_see_the_operations(monkeypatch):
    """Fake tensors, operation counters and wrapper tensors work through the operations a launch would hide."""
    from torch.utils._python_dispatch import TorchDispatchMode

    class Mode(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            return func(*args, **(kwargs or {}))

    class Wrapped(torch.Tensor):
        pass

    monkeypatch.setattr(decode_ops, "_on_cuda", lambda t: True)
    x, rows = torch.zeros(2, 400, 8, dtype=torch.bfloat16), 800
    assert decode_ops._rows_ok(x, rows, x, torch.nn.Parameter(x, requires_grad=False))
    assert not decode_ops._rows_ok(x, rows, x.as_subclass(Wrapped)) and not decode_ops._rows_ok(x.as_subclass(Wrapped), rows)
    with Mode():
        assert not decode_ops._rows_ok(x, rows, x)
    assert decode_ops._rows_ok(x, rows, x)


def test_operands_a_launch_would_read_past_are_left_to_torch(monkeypatch):
    """Tables and weights that torch broadcasts or refuses: a launch would read a full row of them through a pointer."""
    launches = []
    monkeypatch.setattr(decode_ops, "_on_cuda", lambda t: True)
    for name in STAND_INS:
        monkeypatch.setattr(decode_ops, name, lambda *a, name=name: launches.append(name) or STAND_INS[name](*a))
    patched, _ = _models("cpu")
    from transformers.models.llama import modeling_llama as ml

    B, T, hd = 2, 300, 64
    q = torch.randn(B, T, 4, hd).to(torch.bfloat16).transpose(1, 2)
    cos, sin = torch.randn(1, T, hd).to(torch.bfloat16), torch.randn(1, T, hd).to(torch.bfloat16)
    ml.apply_rotary_pos_emb(q, q, cos, sin)
    assert launches == ["rope"]
    for c, s in ((cos[:, :1], sin[:, :1]), (cos, sin[:, :1]), (cos[..., :1], sin[..., :1]), (cos, sin.float())):
        out = ml.apply_rotary_pos_emb(q, q, c.contiguous(), s.contiguous())
        assert out[0].shape == q.shape and launches == ["rope"]
    norm, x = patched.model.norm, torch.randn(B, T, 256).to(torch.bfloat16)
    launches.clear()
    norm(x)
    assert launches == ["rmsnorm"] and decode_ops._add_norm_ok(x, x, norm)
    for w in (torch.ones(1), torch.ones(1).expand(256)):
        norm.weight = torch.nn.Parameter(w.to(torch.bfloat16) if w.is_contiguous() else torch.ones(1, dtype=torch.bfloat16).expand(256), requires_grad=False)
        assert norm(x).shape == x.shape and launches == ["rmsnorm"] and not decode_ops._add_norm_ok(x, x, norm)
