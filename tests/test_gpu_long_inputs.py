"""The fused elementwise kernels on inputs of more than 512 token rows, and where they must not be used."""
from __future__ import annotations

import pytest
import torch

from ade_b200 import decode_ops, synth

pytestmark = pytest.mark.gpu
DEV = "cuda"


# 16-byte pieces (hd 128, 32), element by element (hd 24; a shifted projection), more elements than one round of the grid
@pytest.mark.parametrize("B,T,h,hd,shift", [(2, 700, 8, 128, 0), (1, 1030, 3, 32, 0), (1, 600, 2, 24, 0), (1, 520, 4, 64, 2)])
def test_rope_and_silu_bit_exact(B, T, h, hd, shift):
    g = torch.Generator().manual_seed(T)
    row = 2 * h * hd + 8
    buf = torch.randn(B * T * row + 16, generator=g).to(torch.bfloat16).to(DEV)
    y = buf[shift:shift + B * T * row].view(B, T, row)
    q, k = y[..., :h * hd].view(B, T, h, hd).transpose(1, 2), y[..., h * hd:2 * h * hd].view(B, T, h, hd).transpose(1, 2)
    ang = torch.rand(1, T, hd, generator=g) * 6.28
    cos, sin = ang.cos().to(torch.bfloat16).to(DEV), ang.sin().to(torch.bfloat16).to(DEV)
    rot = lambda t: torch.cat((-t[..., hd // 2:], t[..., :hd // 2]), dim=-1)
    want = [(t * cos.unsqueeze(1)) + (rot(t) * sin.unsqueeze(1)) for t in (q, k)]
    got = decode_ops.rope(q, k, cos, sin)
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
    gate, up = y[..., :h * hd], y[..., h * hd:2 * h * hd]
    assert torch.equal(decode_ops.silu_mul(gate, up), torch.nn.functional.silu(gate) * up)


def test_long_inputs_fused_only_without_gradients():
    """600 token rows: the patched model launches the fused kernels under no_grad and gives the original's logits; with gradients
    enabled it stays differentiable down to the embeddings."""
    model, _, _ = synth.synthetic_llama("tiny", layers=2, seed=3, device=DEV, vocab=512, fused_ops=False)
    ids = torch.randint(0, 512, (2, 300), device=DEV)
    with torch.no_grad():
        want = model(input_ids=ids, use_cache=False).logits.float()
        decode_ops.enable_fused_decode_ops(model)
        calls = []
        original = decode_ops.rmsnorm
        decode_ops.rmsnorm = lambda *a: calls.append(1) or original(*a)
        try:
            got = model(input_ids=ids, use_cache=False).logits.float()
        finally:
            decode_ops.rmsnorm = original
    assert calls
    assert float((got - want).norm() / want.norm()) < 2e-2
    emb = model.get_input_embeddings()(ids).detach().requires_grad_(True)
    model(inputs_embeds=emb, use_cache=False).logits.float().square().mean().backward()
    assert emb.grad is not None and float(emb.grad.abs().sum()) > 0
