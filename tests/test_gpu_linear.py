"""The tensor-core module kernel (`ade_b200_linear`: base GEMM and delta in one launch, up to 128 token rows) against the CPU oracle."""
from __future__ import annotations

import pytest
import torch

from ade_b200 import _lib, kernels, serving, synth
from oracle import oracle as O

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _case(M, N, r, T):
    tp = synth.random_packed(M, N, r, M + N + T)
    W, x = synth.base_weight(M, N, M + 1), synth.activations(T, N, T + 2)
    return tp, W, x


# one row, one slice per SM and fewer rows than SMs; ragged token counts around the multiples of 16; ragged slices; the highest rank;
# two and three slices per SM (19000 and 38000 rows); the widest token range
@pytest.mark.parametrize("M,N,r,T", [(1, 128, 128, 1), (100, 256, 512, 17), (129, 128, 256, 128), (500, 1024, 128, 33), (1000, 4096, 384, 20),
                                     (4096, 2048, 640, 100), (301, 4096, 1024, 64), (256, 384, 2048, 47), (19000, 128, 256, 40),
                                     (38000, 128, 128, 128), (2050, 1152, 896, 16)])
def test_linear_matches_oracle(M, N, r, T):
    tp, W, x = _case(M, N, r, T)
    p4 = kernels.pack_int4(tp, device=DEV)
    y = kernels.linear_forward(x.to(DEV), p4, W.to(DEV))
    y2 = kernels.linear_forward(x.to(DEV), p4, W.to(DEV))
    torch.cuda.synchronize()
    kernels.check_factored_status(DEV)
    assert torch.equal(y, y2), "two runs differ"
    ref = O.factored_apply(x.view(torch.uint16).numpy(), W.view(torch.uint16).numpy(), O.packed_from_torch(tp))
    err, cos = O.parity(y.float().cpu().numpy(), ref)
    assert err <= 1e-2 and cos >= 0.9999, (err, cos)


@pytest.mark.parametrize("T", [8, 9, 16])
def test_tall_fused_group(T):
    """A group of 16500 rows, on both sides of the line at 8 tokens, against its members alone: the same float32 sums in another
    order, so up to the last bf16 bit (2^-8 of the value, and of the row's terms where they cancel)."""
    N = 128
    mods = []
    for M, r in ((7700, 256), (300, 384), (8500, 128)):
        tp, W, x = _case(M, N, r, T)
        mods.append(serving.ADEKernelLinear(W, tp).to(DEV))
    xd = x.to(DEV)
    alone = [m(xd) for m in mods]
    group = serving.FusedADEGroup(mods)
    assert group.p4["blocks"] is not None
    for a, m in zip(alone, mods):
        y = m(xd)
        assert torch.all((y.float() - a.float()).abs() <= 2.0 ** -7 * (a.float().abs() + a.float().abs().mean()))
    torch.cuda.synchronize()
    kernels.check_factored_status(DEV)


# both ways U^ h is prepared (64 / 65 tokens), one to three slices per SM, ragged rows, the highest rank, fewer rows than SMs
@pytest.mark.parametrize("M,N,r,T", [(5000, 256, 896, 33), (5000, 256, 896, 64), (129, 128, 256, 65), (300, 1024, 2048, 100), (4097, 384, 1024, 47),
                                     (19000, 128, 256, 40), (38000, 128, 128, 128), (1, 128, 128, 128)])
def test_supplied_base_term(M, N, r, T):
    tp, W, x = _case(M, N, r, T)
    assert _lib.load().ade_b200_linear_preferred(T, M, r) == 1
    p4, xd = kernels.pack_int4(tp, device=DEV), x.to(DEV)
    yd = torch.nn.functional.linear(xd, W.to(DEV))
    y, y2 = kernels.decode_forward_packed(xd, yd, p4), kernels.decode_forward_packed(xd, yd, p4)
    torch.cuda.synchronize()
    kernels.check_factored_status(DEV)
    assert torch.equal(y, y2), "two runs differ"
    ref = O.factored_apply(x.view(torch.uint16).numpy(), W.view(torch.uint16).numpy(), O.packed_from_torch(tp))
    err, cos = O.parity(y.float().cpu().numpy(), ref)
    assert err <= 1e-2 and cos >= 0.9999, (err, cos)


def test_linear_wait_expires_and_recovers():
    """Nobody reports h: every CTA's wait runs out, the launch still ends, the status word says so, the next call is right."""
    M, N, r, T = 512, 1024, 256, 40
    tp, W, x = _case(M, N, r, T)
    p4, W, x = kernels.pack_int4(tp, device=DEV), W.to(DEV), x.to(DEV)
    good = kernels.linear_forward(x, p4, W)
    torch.cuda.synchronize()
    _lib.set_option(_lib.OPT_WAIT_LIMIT_CYCLES, 400_000)
    _lib.set_option(_lib.OPT_DROP_SIGNALS, 1)
    try:
        kernels.linear_forward(x, p4, W)
        torch.cuda.synchronize()
        assert kernels.factored_status(DEV, T, r) == 1
        with pytest.raises(_lib.AdeKernelError):
            kernels.check_factored_status(DEV)
    finally:
        _lib.set_option(_lib.OPT_DROP_SIGNALS, 0)
        _lib.set_option(_lib.OPT_WAIT_LIMIT_CYCLES, 0)
        kernels.reset_factored_scratch(DEV)
    again = kernels.linear_forward(x, p4, W)
    torch.cuda.synchronize()
    assert kernels.factored_status(DEV, T, r) == 0 and torch.equal(again, good)


def test_linear_argument_checks():
    tp, W, x = _case(256, 256, 128, 20)
    p4 = kernels.pack_int4(tp, device=DEV)
    with pytest.raises(ValueError):
        kernels.linear_forward(x.to(DEV), p4, W.to(DEV).t())
    with pytest.raises(ValueError):
        kernels.linear_forward(x.float().to(DEV), p4, W.to(DEV))
    with pytest.raises(_lib.AdeKernelError):
        kernels.linear_forward(torch.zeros(129, 256, dtype=torch.bfloat16, device=DEV), p4, W.to(DEV))


@pytest.mark.parametrize("M,T", [(16384, 8), (16384, 9), (16383, 9), (16384, 17), (300, 16), (300, 17), (300, 64), (300, 65)])
def test_module_dispatch_edges(M, T):
    """Both sides of the lines between the two kernels, through the module."""
    N, r = 128, 128
    tp, W, x = _case(M, N, r, T)
    y = serving.ADEKernelLinear(W, tp).to(DEV)(x.to(DEV))
    torch.cuda.synchronize()
    kernels.check_factored_status(DEV)
    ref = O.factored_apply(x.view(torch.uint16).numpy(), W.view(torch.uint16).numpy(), O.packed_from_torch(tp))
    err, cos = O.parity(y.float().cpu().numpy(), ref)
    assert err <= 1e-2 and cos >= 0.9999, (err, cos)


def _direct(entry, x, p4, y=None, W=None):
    """One of the two kernels by its C entry, whatever the dispatch says."""
    import ctypes

    lib, (T, M, r) = _lib.load(), (x.shape[0], p4["M"], p4["r"])
    out = torch.empty(T, M, dtype=torch.bfloat16, device=DEV)
    scratch = torch.zeros(lib.ade_b200_factored_scratch_bytes(T, r), dtype=torch.uint8, device=DEV)
    args = [ctypes.byref(kernels._cdelta(p4)), x.data_ptr(), None if y is None else y.data_ptr(), None if W is None else W.data_ptr(),
            out.data_ptr(), scratch.data_ptr(), scratch.numel()]
    work = torch.empty(lib.ade_b200_linear_workspace_bytes(T, M, r), dtype=torch.uint8, device=DEV)
    if entry == "linear":
        args += [work.data_ptr(), work.numel()]
    assert getattr(lib, f"ade_b200_{entry}")(*args, T, torch.cuda.current_stream().cuda_stream) == 0
    torch.cuda.synchronize()
    return out


# both sides of every line of the rule for calls with y_dense: tokens, rows times rank, rows per SM, h in shared memory, columns and rank
@pytest.mark.parametrize("M,N,r,T,linear", [(31250, 128, 128, 32, 0), (31250, 128, 128, 33, 1), (31249, 128, 128, 33, 0), (31249, 128, 128, 65, 1),
                                            (4736, 384, 384, 65, 0), (4737, 384, 384, 65, 1), (4736, 128, 256, 128, 1), (600, 384, 1024, 87, 0),
                                            (600, 384, 1024, 90, 1), (500, 1152, 768, 80, 1), (500, 1024, 768, 80, 0), (500, 1152, 896, 80, 0),
                                            (300, 4096, 896, 66, 1), (2048, 8192, 128, 65, 1), (2049, 8192, 128, 65, 0), (4000, 8192, 1024, 40, 1), (4000, 8064, 1024, 40, 0), (3200, 6144, 1280, 34, 1)])
def test_supplied_base_term_takes_the_kernel_of_the_rule(M, N, r, T, linear):
    assert _lib.load().ade_b200_linear_faster(T, M, N, r, 0) == linear
    p4 = kernels.pack_int4(synth.random_packed(M, N, r, M + T, DEV, on_device=True))
    x, y = synth.activations(T, N, 1).to(DEV), synth.activations(T, M, 2).to(DEV)
    by = {e: _direct(e, x, p4, y) for e in ("factored", "linear")}
    assert torch.equal(kernels.decode_forward_packed(x, y, p4), by["linear" if linear else "factored"])
    err, cos = O.parity(by["linear"].float().cpu().numpy(), by["factored"].float().cpu().numpy())
    assert err <= 1e-2 and cos >= 0.9999, (err, cos)


# the rule for calls with the base weight, one block and two: rows, tokens, ranks of a row against columns, and where h takes the third FIFO
# stage (with four columns for each rank of a row)
@pytest.mark.parametrize("M,N,r,T,blocks,linear", [(16383, 128, 128, 9, 1, 0), (16384, 128, 128, 8, 1, 0), (16384, 128, 128, 9, 1, 1), (16384, 128, 256, 9, 2, 1),
                                                   (16384, 128, 256, 9, 1, 0), (16384, 3072, 256, 16, 1, 1), (16384, 2944, 256, 16, 1, 0),
                                                   (16384, 3072, 512, 16, 2, 1), (22016, 2176, 1024, 15, 2, 0), (22016, 2176, 1024, 16, 2, 1),
                                                   (22016, 2176, 1024, 16, 1, 0), (22016, 2048, 1024, 16, 2, 0)])
def test_module_takes_the_kernel_of_the_rule(M, N, r, T, blocks, linear):
    assert _lib.load().ade_b200_linear_faster(T, M, N, r, blocks) == linear
    p4 = kernels.pack_int4(synth.random_packed(M, N, r, M + T, DEV, on_device=True))
    if blocks == 2:
        p4["blocks"] = [(0, 0), (M // 2, r // 256), (M, r // 128)]
        p4["us"][:M // 2, r // 256:], p4["us"][M // 2:, :r // 256] = 0, 0
    x, W = synth.activations(T, N, 1).to(DEV), synth.base_weight(M, N, 2).to(DEV)
    by = {e: _direct(e, x, p4, W=W) for e in ("factored", "linear")}
    assert torch.equal(kernels.module_forward(x, p4, W), by["linear" if linear else "factored"])
    err, cos = O.parity(by["linear"].float().cpu().numpy(), by["factored"].float().cpu().numpy())
    assert err <= 1e-2 and cos >= 0.9999, (err, cos)


# the form with y_dense on both ways U^ h is prepared (64 / 65 tokens), one to three slices per SM, ragged rows, the highest rank, fewer rows
# than SMs, whatever the dispatch would take
@pytest.mark.parametrize("M,N,r,T", [(5000, 256, 896, 17), (4097, 384, 1024, 47), (129, 128, 256, 64), (129, 128, 256, 65), (300, 1024, 2048, 100),
                                     (19000, 128, 256, 40), (38000, 128, 128, 128), (1, 128, 128, 1)])
def test_supplied_base_term_by_its_entry(M, N, r, T):
    tp, W, x = _case(M, N, r, T)
    p4, xd = kernels.pack_int4(tp, device=DEV), x.to(DEV)
    y = _direct("linear", xd, p4, torch.nn.functional.linear(xd, W.to(DEV)))
    ref = O.factored_apply(x.view(torch.uint16).numpy(), W.view(torch.uint16).numpy(), O.packed_from_torch(tp))
    err, cos = O.parity(y.float().cpu().numpy(), ref)
    assert err <= 1e-2 and cos >= 0.9999, (err, cos)
