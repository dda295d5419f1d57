"""State of a delta module that a program changes after it was built: tensors swapped, parametrized or written in place."""
from __future__ import annotations

import pytest
import torch
from torch import nn
from torch.nn.utils import parametrize

from ade_b200 import serving, synth

M, N, R = 256, 128, 128


def _module(seed=0):
    return serving.ADEKernelLinear(synth.base_weight(M, N, seed), synth.random_packed(M, N, R, seed + 1))


class _Double(nn.Module):
    def forward(self, w):
        return w * 2


@pytest.mark.parametrize("tokens", [3, 16, 40, 128])
@pytest.mark.parametrize("how", ["buffer", "parameter", "parametrized", "codes_as_parameter"])
def test_weight_need_not_be_a_buffer(monkeypatch, tokens, how):
    """What forward hands to the kernels is the attribute, whatever the module keeps it as."""
    seen = []
    monkeypatch.setattr(serving, "module_forward", lambda x, p4, w: seen.append((p4, w)) or torch.zeros(x.shape[0], M, dtype=torch.bfloat16))
    mod = _module()
    mod(torch.zeros(1, N, dtype=torch.bfloat16))
    seen.clear()
    want = mod.weight.clone()
    if how == "parameter":
        mod.weight = nn.Parameter(want * 3, requires_grad=False)
        want = want * 3
    elif how == "parametrized":
        parametrize.register_parametrization(mod, "weight", _Double())
        want = want * 2
    elif how == "codes_as_parameter":
        mod.p4_uq = nn.Parameter(mod.p4_uq.clone(), requires_grad=False)
    assert mod(torch.zeros(tokens, N, dtype=torch.bfloat16)).shape == (tokens, M)
    (p4, w), = seen
    assert torch.equal(w, want) and p4["uq"].data_ptr() == mod.p4_uq.data_ptr()


def _fields(src, dst, how):
    """Give module `dst` the delta of module `src`."""
    state = {k: v.clone() for k, v in src.state_dict().items()}
    if how == "copy":
        for k, v in state.items():
            dst.get_buffer(k).copy_(v)
    else:
        dst.load_state_dict(state, assign=how == "assign")


@pytest.mark.parametrize("inference", ["never", "always", "first call"])
@pytest.mark.parametrize("how", ["copy", "load", "assign"])
def test_expanded_operands_follow_the_codes(monkeypatch, how, inference):
    """The operands kept for long inputs are made again when the codes change in place or are replaced, and only then."""
    made = []

    def expand(p4):
        made.append(1)
        return p4["uq"].clone(), p4["vq"].clone()

    monkeypatch.setattr(serving, "expand_codes_f8", expand)
    with torch.inference_mode(inference == "always"):
        mod, other = _module(0), _module(5)
    with torch.inference_mode(inference != "never"):
        first = mod._expanded()
    if inference == "always":
        assert first is None                                              # a change could not be noticed
        return
    assert mod._expanded() is first and len(made) == 1
    _fields(other, mod, how)
    u8, v8 = mod._expanded()
    assert len(made) == 2 and torch.equal(u8, other.p4_uq) and torch.equal(v8, other.p4_vq)
    assert mod._expanded()[0] is u8 and len(made) == 2


@pytest.mark.gpu
@pytest.mark.parametrize("how", ["copy", "load", "assign"])
def test_another_delta_in_place(how):
    """Long and short inputs of a module that got another delta equal those of a module built with it, bit for bit."""
    g = torch.Generator().manual_seed(7)
    xs = [torch.randn(t, N, generator=g).to(torch.bfloat16).cuda() for t in (200, 5, 100)]
    mod, other = _module(0).cuda(), _module(5).cuda()
    for x in xs:
        mod(x)
    _fields(other, mod, how)
    for x in xs:
        assert torch.equal(mod(x), other(x))
