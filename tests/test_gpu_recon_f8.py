"""Reconstruction from e4m3 operands (float32 accumulators): the same bits as the integer kernels."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from ade_b200 import _lib, kernels, synth
from oracle import oracle as O

pytestmark = pytest.mark.gpu
DEV = "cuda"


# one to eight groups (both configurations and the unrolled one of four groups), ragged rows, several strips and tiles per CTA
@pytest.mark.parametrize("M,N,r", [(1, 128, 128), (129, 384, 256), (100, 256, 512), (3000, 2048, 512), (2100, 1920, 384), (1024, 1152, 640),
                                   (384, 128, 1024), (2500, 2304, 896)])
def test_recon_f8_bit_exact(M, N, r):
    tp, W = synth.random_packed(M, N, r, M + N + r), synth.base_weight(M, N, 3)
    p4 = kernels.pack_int4(tp, device=DEV)
    Wd = W.to(DEV)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    out = kernels.recon_int4(p4, Wd, status=status, expanded=kernels.expand_codes_f8(p4))
    one_shot = kernels.recon_int4(p4, Wd)
    integer = kernels.recon_int4(p4, Wd, expanded=kernels.expand_codes(p4))
    torch.cuda.synchronize()
    assert int(status.item()) == 0
    _, merged = O.reconstruct(O.packed_from_torch(tp), base_bits=W.view(torch.uint16).numpy())
    assert np.array_equal(out.cpu().view(torch.uint16).numpy(), merged)
    assert torch.equal(out, one_shot) and torch.equal(out, integer)


def test_expand_codes_f8_values():
    tp = synth.random_packed(200, 256, 256, 4)
    u8, v8 = kernels.expand_codes_f8(kernels.pack_int4(tp, device=DEV))
    assert u8.dtype == torch.float8_e4m3fn and u8.shape == (200, 256) and v8.shape == (256, 256)
    u = tp["U_codes"].float() - tp["U_zero"].float().repeat_interleave(128, 1)
    v = (tp["Vt_codes"].float() - tp["Vt_zero"].float().repeat_interleave(128, 0)).t()
    assert torch.equal(u8.float().cpu(), u) and torch.equal(v8.float().cpu(), v)


@pytest.mark.parametrize("high,cancel", [(15, False), (15, True), (14, False)])
def test_accumulators_are_exact(high, cancel):
    """Group products up to 128 * 225 = 28 800 with every bit visible: scales of 1 and a base of -bf16(P) leave the part of P that
    bf16 cannot hold.  `cancel`: large partial sums of both signs."""
    M, N, r = 256, 384, 128
    g = torch.Generator().manual_seed(high + cancel)
    uc = torch.randint(high - 2, high + 1, (M, r), generator=g)
    vc = torch.randint(high - 2, high + 1, (r, N), generator=g)
    vz = torch.zeros(1, N)
    if cancel:
        vc[64:] = torch.randint(0, 2, (64, N), generator=g)
        vz = torch.full((1, N), 7.0)
    tp = {"U_codes": uc.to(torch.uint8), "Vt_codes": vc.to(torch.uint8), "U_scale": torch.ones(M, 1, dtype=torch.bfloat16),
          "Vt_scale": torch.ones(1, N, dtype=torch.bfloat16), "U_zero": torch.zeros(M, 1, dtype=torch.bfloat16), "Vt_zero": vz.to(torch.bfloat16)}
    P = uc.double() @ (vc.double() - vz.double())
    W = (-P).to(torch.bfloat16)
    p4 = kernels.pack_int4(tp, device=DEV)
    out = kernels.recon_int4(p4, W.to(DEV), expanded=kernels.expand_codes_f8(p4)).cpu()
    assert torch.equal(out.double(), W.double() + P)


def test_f8_operands_and_dump_are_exclusive():
    p4 = kernels.pack_int4(synth.random_packed(128, 128, 128, 1), device=DEV)
    W = synth.base_weight(128, 128, 2).to(DEV)
    acc = torch.empty(1, 128, 128, dtype=torch.int32, device=DEV)
    with pytest.raises((RuntimeError, _lib.AdeKernelError)):
        kernels.recon_int4(p4, W, dbg_acc=acc, expanded=kernels.expand_codes_f8(p4))


# both configurations and the unrolled one; 446 strips of one tile: every CTA walks three strips or more, so each us table is used a third time
@pytest.mark.parametrize("r", [256, 512, 640])
def test_three_strips_of_one_tile_per_cta(r):
    M, N = 57000, 128
    tp, W = synth.random_packed(M, N, r, r), synth.base_weight(M, N, 3)
    p4, Wd = kernels.pack_int4(tp, device=DEV), W.to(DEV)
    out = kernels.recon_int4(p4, Wd, expanded=kernels.expand_codes_f8(p4))
    torch.cuda.synchronize()
    _, merged = O.reconstruct(O.packed_from_torch(tp), base_bits=W.view(torch.uint16).numpy())
    assert np.array_equal(out.cpu().view(torch.uint16).numpy(), merged)


@pytest.mark.parametrize("pattern", ["uniform", "extremes", "one sign"])
@pytest.mark.parametrize("r,group", [(128, 0), (384, 1), (512, 3), (1024, 0), (1024, 7)])
def test_accumulators_are_exact_in_every_group(r, group, pattern):
    """As above with one group of several looked at (the others have scale 0): codes and zero-points over their whole range, products of 0
    and plus and minus 225, and products of one sign."""
    M, N, ng = 200, 256, r // 128
    g = torch.Generator().manual_seed(r + group)
    uz, vz = torch.randint(0, 16, (M, ng), generator=g), torch.randint(0, 16, (ng, N), generator=g)
    uc, vc = torch.randint(0, 16, (M, r), generator=g), torch.randint(0, 16, (r, N), generator=g)
    if pattern == "extremes":
        uz, vz = torch.randint(0, 2, (M, ng), generator=g) * 15, torch.randint(0, 2, (ng, N), generator=g) * 15
        uc, vc = 15 - uz.repeat_interleave(128, 1), torch.randint(0, 2, (r, N), generator=g) * 15
    elif pattern == "one sign":
        uz, vz = torch.zeros(M, ng), torch.zeros(ng, N)
        uc, vc = torch.randint(11, 16, (M, r), generator=g), torch.randint(11, 16, (r, N), generator=g)
    us, vs = torch.zeros(M, ng), torch.zeros(ng, N)
    us[:, group], vs[group] = 1, 1
    tp = {"U_codes": uc.to(torch.uint8), "Vt_codes": vc.to(torch.uint8), "U_scale": us.to(torch.bfloat16), "Vt_scale": vs.to(torch.bfloat16),
          "U_zero": uz.to(torch.bfloat16), "Vt_zero": vz.to(torch.bfloat16)}
    k = slice(128 * group, 128 * group + 128)
    P = (uc[:, k].double() - uz[:, group:group + 1].double()) @ (vc[k].double() - vz[group:group + 1].double())
    W = (-P).to(torch.bfloat16)                         # 8 of at most 15 bits: the other 7 are what the result shows
    p4 = kernels.pack_int4(tp, device=DEV)
    out = kernels.recon_int4(p4, W.to(DEV), expanded=kernels.expand_codes_f8(p4)).cpu()
    assert torch.equal(out.double(), W.double() + P)
