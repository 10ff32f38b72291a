"""Rows of one warp that differ in where their scores are -inf or near the lowest float32, against float64: every form of the
attention kernel has to give the softmax over the keys that are left, wherever its blocks and parts begin.

The mask travels in one column of the head: q there is a for the rows that are masked and 0 for the others, k there is b for the
keys that are masked and 0 for the others, so a masked score is a * b plus a few units."""
import pytest
import torch

from ditto_b200 import _lib, ops
from tests.test_gpu_attention_split import _close, _reference

pytestmark = pytest.mark.gpu

FORMS = {"narrow": _lib.FLAG_NARROW, "split 2": 2 * _lib.FLAG_SPLIT_UNIT, "split 4": 3 * _lib.FLAG_SPLIT_UNIT,
         "few 1": _lib.FLAG_FEW, "few 2": _lib.FLAG_FEW | 2 * _lib.FLAG_SPLIT_UNIT, "few 4": _lib.FLAG_FEW | 3 * _lib.FLAG_SPLIT_UNIT,
         "whole": _lib.FLAG_SPLIT_UNIT, "one tile": _lib.FLAG_ONE_TILE, "two tiles": _lib.FLAG_TWO_TILES,
         "P via smem": _lib.FLAG_P_VIA_SMEM}
# masked keys of 512: less than a block, whole blocks at the start, in the middle and at the end, whole parts, all but a few
MASKED = ((0, 64), (0, 128), (64, 192), (128, 256), (256, 384), (0, 256), (256, 512), (0, 496), (16, 512))
# a, b, type: a product that overflows float32 to -inf; the lowest values of the two types; large ones that a float32 can tell apart
VALUES = ((1e30, -1e30, torch.bfloat16), (1.0, torch.finfo(torch.bfloat16).min, torch.bfloat16), (1.0, -1e30, torch.bfloat16),
          (1.0, torch.finfo(torch.float16).min, torch.float16))


@pytest.mark.parametrize("a,b,dtype", VALUES)
@pytest.mark.parametrize("form,d", [(f, d) for f in FORMS for d in (64, 128) if d == 64 or f != "narrow"])
def test_rows_masked_apart(form, d, a, b, dtype):
    g = torch.Generator(device="cuda").manual_seed(11)
    M, L = 160, 512
    for scale in (d ** -0.5, 2.0):
        q = torch.randn(1, M, d, generator=g, device="cuda")
        k = torch.randn(1, L, d, generator=g, device="cuda")
        if scale > 1:
            q *= 0.25
        v = torch.randn(1, L, d, generator=g, device="cuda").to(dtype)
        masked_rows = torch.arange(M, device="cuda") % 3 == 1
        q[:, :, 5] = torch.where(masked_rows, a, 0.0)
        q = q.to(dtype)
        for lo, hi in MASKED:
            kk = k.clone()
            kk[:, :, 5] = 0.0
            kk[:, lo:hi, 5] = b
            kk = kk.to(dtype)
            out = ops.bmm_softmax_bmm(q, kk, v, scale=scale, key_layout="LK", flags=FORMS[form])
            _close(out, _reference(q, kk, v, scale), dtype)
    assert ops.device_status() == 0


@pytest.mark.parametrize("form,d", [(f, d) for f in FORMS for d in (64, 128) if d == 64 or f != "narrow"])
def test_row_without_a_finite_score(form, d):
    """0 / 0 as in torch.softmax -- in that row alone."""
    g = torch.Generator(device="cuda").manual_seed(12)
    q = torch.randn(1, 128, d, generator=g, device="cuda")
    k = torch.randn(1, 512, d, generator=g, device="cuda")
    q[:, :, 5] = torch.where(torch.arange(128, device="cuda") == 40, 1e30, 0.0)
    k[:, :, 5] = -1e30
    q, k = q.bfloat16(), k.bfloat16()
    v = torch.randn(1, 512, d, generator=g, device="cuda").bfloat16()
    out = ops.bmm_softmax_bmm(q, k, v, scale=0.125, key_layout="LK", flags=FORMS[form])
    assert out[:, 40].isnan().all()
    keep = [i for i in range(128) if i != 40]
    _close(out[:, keep], _reference(q[:, keep], k, v, 0.125), torch.bfloat16)


@pytest.mark.parametrize("form,d", [(f, d) for f in FORMS for d in (64, 128) if d == 64 or f != "narrow"])
def test_references_that_rounding_moves(form, d):
    """Scores of about 2^31 one unit in the last place apart, at scales that make an exponent of 2 of them about 2^32: rounding the
    reference's alone moves a row's exponents by up to 256, above what float32 holds.  A row may be NaN then, or what its largest
    score says (the next one weighs 2^-257 of it); weights that have run over into the sign or into small numbers it may not show."""
    g = torch.Generator(device="cuda").manual_seed(13)
    M, L = 128, 128
    q = torch.zeros(1, M, d, device="cuda")
    q[:, :, :2] = 1.0
    v = torch.randn(1, L, d, generator=g, device="cuda").bfloat16()
    for first in list(range(16)) + [47, 127]:
        k = torch.zeros(1, L, d, device="cuda")
        k[:, [first, 20], 0] = 255.0 * 2 ** 23                 # (with the second column 24 bits: exact in float32)
        k[:, first, 1], k[:, 20, 1] = 256.0, 128.0
        for step in range(24):
            scale = 1.4 * (1 + step / 2000)
            c = torch.tensor(scale, dtype=torch.float32) * torch.tensor(1.4426950408889634, dtype=torch.float32)
            score = torch.tensor(255.0 * 2 ** 23 + 256.0)
            moved = (score.double() * c.double() - (score * c).double()).item()
            assert (score * c).item() > 2 ** 32 and abs(moved) <= 256
            if 125 < moved < 128.1:                            # 1 / sum is below the smallest normal number
                continue
            out = ops.bmm_softmax_bmm(q.bfloat16(), k.bfloat16(), v, scale=scale, key_layout="LK", flags=FORMS[form])
            want = v[:, first:first + 1].expand(1, M, d)
            rows = out.isnan().all(dim=-1)
            assert not out.isnan().any() or rows.all(), (first, scale, moved)
            assert rows.all() or (out.double() - want.double()).abs().max() <= 2 ** -7 * want.abs().max(), (first, scale, moved)
    assert ops.device_status() == 0
