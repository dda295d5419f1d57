"""State of a delta module that a program changes after it was built: tensors swapped, parametrized or written in place."""
from __future__ import annotations

import copy

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


def _group(seeds):
    return serving.FusedADEGroup([_module(s) for s in seeds])


@pytest.mark.parametrize("how", ["copy", "load", "assign"])
@pytest.mark.parametrize("member", [0, 1])
def test_group_follows_its_members(monkeypatch, how, member):
    """A delta written into a member after the group was built is what the group's launch uses, at the same addresses."""
    seen = []
    monkeypatch.setattr(serving, "module_forward", lambda x, p4, w: seen.append((p4, w)) or torch.zeros(x.shape[0], w.shape[0], dtype=torch.bfloat16))
    group, other, x = _group((0, 3)), _module(9), torch.zeros(4, N, dtype=torch.bfloat16)
    other.weight.copy_(group.members[member].weight)
    addresses = {k: group.p4[k].data_ptr() for k in serving.STORED_KEYS}
    [m(x) for m in group.members]
    assert len(seen) == 1 and seen[0][0] is group.p4
    if how == "assign":
        keep = group.members[member].weight
        _fields(other, group.members[member], how)
        group.members[member].weight = keep                       # the base weight stays a view of the group's
    else:
        _fields(other, group.members[member], how)
    want = serving.FusedADEGroup([_module(9 if i == member else s) for i, s in enumerate((0, 3))]).p4
    [m(x.clone()) for m in group.members[:1]]
    assert seen[-1][0] is group.p4
    for k in serving.STORED_KEYS:
        assert torch.equal(group.p4[k], want[k]) and group.p4[k].data_ptr() == addresses[k], k


@pytest.mark.parametrize("member", [0, 1])
def test_group_dissolves_when_a_weight_is_kept_elsewhere(monkeypatch, member):
    seen = []
    monkeypatch.setattr(serving, "module_forward", lambda x, p4, w: seen.append(w) or torch.zeros(x.shape[0], w.shape[0], dtype=torch.bfloat16))
    group, x = _group((0, 3)), torch.zeros(4, N, dtype=torch.bfloat16)
    mods = group.members
    mods[member].weight = nn.Parameter(mods[member].weight * 2, requires_grad=False)
    for m in mods:
        assert m(x).shape == (4, M)
    assert not group.refresh() and all(m._group is None for m in mods)
    assert [w.shape[0] for w in seen] == [M, M] and torch.equal(seen[member], mods[member].weight)


@pytest.mark.gpu
def test_captured_generation_follows_another_delta():
    """Another delta written into the modules after a step was captured: the next generation, whose prompt is longer than a group serves,
    gives the tokens of groups built from it."""
    from ade_b200 import kernels

    model = synth.synthetic_llama("tiny", layers=2, seed=1, vocab=512)[0]
    ids = torch.randint(0, 512, (1, 30), generator=torch.Generator().manual_seed(4)).cuda()
    dec = serving.GreedyGraphDecoder(model)
    before = dec.generate(ids, 12)
    mods = [m for m in model.modules() if isinstance(m, serving.ADEKernelLinear)]
    for i, m in enumerate(mods):
        packed = synth.random_packed(*m._dims, 50 + i)
        packed["U_scale"] *= 20
        for k, v in kernels.pack_int4(packed).items():
            if k in serving.STORED_KEYS:
                m.get_buffer(f"p4_{k}").copy_(v)
    got = dec.generate(ids, 12)
    for m in mods:
        if m._group is not None:
            m._group[0].release()
    assert serving.fuse_kernel_linears(model) == 4
    want = serving.GreedyGraphDecoder(model).generate(ids, 12, use_graph=False)
    assert torch.equal(got, want) and not torch.equal(got, before)


def test_group_members_serve_inference_tensors(monkeypatch):
    """Under torch.inference_mode a tensor has no version counter: the members launch for themselves."""
    seen = []
    monkeypatch.setattr(serving, "module_forward", lambda x, p4, w: seen.append(w) or torch.zeros(x.shape[0], w.shape[0], dtype=torch.bfloat16))
    group = _group((0, 3))
    with torch.inference_mode():
        x = torch.zeros(4, N, dtype=torch.bfloat16)
        for m in group.members:
            assert m(x).shape == (4, M)
    assert [w.shape[0] for w in seen] == [M, M] and group.refresh()


def test_expanded_operands_made_during_a_capture_are_not_kept(monkeypatch):
    """What a capturing stream makes holds nothing before the graph runs, and its memory is the graph's."""
    monkeypatch.setattr(serving, "expand_codes_f8", lambda p4: (p4["uq"].clone(), p4["vq"].clone()))
    mod, capturing = _module(0), [True]
    monkeypatch.setattr(serving, "_capturing", lambda t: capturing[0], raising=False)
    first = mod._expanded()
    assert mod._x8 is None and mod._expanded()[0] is not first[0]
    capturing[0] = False
    kept = mod._expanded()
    capturing[0] = True
    assert mod._expanded() is kept
    twin = copy.deepcopy(mod)
    assert twin._x8 is None and torch.equal(twin._expanded()[0], kept[0])


@pytest.mark.gpu
def test_expanded_operands_are_waited_for_on_another_stream():
    """Two streams, the first use on one of them behind queued work: the other waits until the operands are there."""
    mod = _module(0).cuda()
    x = torch.randn(200, N, generator=torch.Generator().manual_seed(1)).to(torch.bfloat16).cuda()
    want = _module(0).cuda()(x)
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    torch.cuda._sleep(100_000_000)
    a = mod(x)
    with torch.cuda.stream(side):
        b = mod(x)
    torch.cuda.synchronize()
    assert torch.equal(a, want) and torch.equal(b, want)


@pytest.mark.gpu
def test_dimensions_of_a_stored_form_may_be_tensors():
    """As a file's loader may leave them: one scratch buffer serves repeated calls."""
    from ade_b200 import kernels

    mod = _module(0).cuda()
    p4 = {k: v if k in serving.STORED_KEYS else torch.tensor(v) for k, v in mod._stored_form().items()}
    x = torch.randn(24, N, generator=torch.Generator().manual_seed(1)).to(torch.bfloat16).cuda()
    want = mod(x)
    buffers = len(kernels._scratch)
    for _ in range(3):
        assert torch.equal(kernels.module_forward(x, p4, mod.weight), want)
    assert len(kernels._scratch) == buffers
