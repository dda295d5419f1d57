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
