"""The reconstruction kernels that unpack codes inside, launched many times: every launch gives the same bits.

The raw-code ring is refilled by copies while the unpack warps work; a slot handed back before its reads were over gave one tile column
the codes of the slot's next item in one launch of some two hundred."""
from __future__ import annotations

import pytest
import torch

from ade_b200 import kernels, synth

pytestmark = pytest.mark.gpu
DEV = "cuda"


# two, four and eight groups: both configurations of the strip kernel, with and without the accumulator dump
@pytest.mark.parametrize("M,N,r,launches", [(13824, 5120, 256, 300), (5120, 5120, 512, 300), (5120, 5120, 1024, 600)])
def test_every_launch_gives_the_same_bits(M, N, r, launches):
    ng = r // 128
    tp = synth.random_packed(M, N, r, 3 * r + M, DEV, on_device=True)
    p4, W = kernels.pack_int4(tp), torch.zeros(M, N, dtype=torch.bfloat16, device=DEV)
    u = (tp["U_codes"].view(M, ng, 128).float() - tp["U_zero"].float().unsqueeze(2))
    v = (tp["Vt_codes"].view(ng, 128, N).float() - tp["Vt_zero"].float().unsqueeze(1))
    want = torch.stack([(u[:, g].double() @ v[g].double()).to(torch.int32) for g in range(ng)])
    merged = kernels.recon_int4(p4, W, expanded=kernels.expand_codes(p4))
    acc = torch.empty_like(want)
    wrong = torch.zeros((), dtype=torch.int64, device=DEV)
    for _ in range(launches):
        out = kernels.recon_int4(p4, W, dbg_acc=acc)
        wrong += (acc != want).sum() + (out != merged).sum()
    plain = torch.empty_like(W)
    import ctypes

    from ade_b200 import _lib

    d, st = ctypes.byref(kernels._cdelta(p4)), torch.cuda.current_stream().cuda_stream
    for _ in range(launches):
        assert _lib.load().ade_b200_recon(d, W.data_ptr(), plain.data_ptr(), None, None, st) == 0
        wrong += (plain != merged).sum()
    assert int(wrong) == 0
