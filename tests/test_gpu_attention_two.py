"""The kernel for few items in the form of which two CTAs fit an SM at head dimension 128 (more than 148 tiles), against float64: one and several tiles a
sequence, ragged rows and keys, widths below 128 and apart, one to many blocks, both layouts and types, chains without a softmax, rows whose
scores are masked; and what the rule picks it for."""
import pytest
import torch

from ditto_b200 import ops
from tests.test_gpu_attention_masked_rows import MASKED, VALUES
from tests.test_gpu_attention_short import _launched, _operands
from tests.test_gpu_attention_split import _close, _reference

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("layout", ["LK", "KL"])
@pytest.mark.parametrize("b,M,N,K,L", [
    (150, 128, 128, 128, 16), (160, 16, 80, 80, 272), (149, 112, 16, 128, 128), (300, 128, 128, 96, 400), (75, 208, 80, 80, 208),
    (148, 256, 112, 128, 384), (40, 512, 128, 112, 512), (30, 528, 128, 80, 448), (450, 64, 128, 128, 1040), (600, 128, 96, 96, 304)])
def test_softmax(b, M, N, K, L, layout, dtype):
    q, k, v = _operands(b, M, N, K, L, dtype, b + L)
    keys = k if layout == "LK" else k.transpose(1, 2).contiguous()
    scale = 2 * K ** -0.5
    out = torch.full((b, M, N), float("nan"), dtype=dtype, device="cuda")
    got = _launched(lambda: ops.bmm_softmax_bmm(q, keys, v, out, scale=scale, key_layout=layout))
    assert got == ("few", b * ((M + 127) // 128))
    want = out.clone()
    ops.bmm_softmax_bmm(q, keys, v, out, scale=scale, key_layout=layout)
    assert ops.device_status() == 0 and torch.equal(out, want)
    for i in range(0, b, 37):
        _close(out[i:i + 1], _reference(q[i:i + 1], k[i:i + 1], v[i:i + 1], scale), dtype)


@pytest.mark.parametrize("act", ["identity", "relu"])
@pytest.mark.parametrize("layout", ["IO", "OI"])
@pytest.mark.parametrize("b,M,N,K,L", [(150, 128, 128, 128, 80), (300, 16, 16, 96, 528), (75, 256, 128, 80, 2064), (180, 208, 80, 128, 528)])
def test_chains(act, layout, b, M, N, K, L):
    g = torch.Generator(device="cuda").manual_seed(M + L)
    x = torch.randn(b, M, K, generator=g, device="cuda").half()
    w1 = (torch.randn(b, K, L, generator=g, device="cuda") * K ** -0.5).half()
    w2 = (torch.randn(b, L, N, generator=g, device="cuda") * L ** -0.5).half()
    ws = (w1, w2) if layout == "IO" else (w1.transpose(1, 2).contiguous(), w2.transpose(1, 2).contiguous())
    out = torch.full((b, M, N), float("nan"), dtype=torch.float16, device="cuda")
    got = _launched(lambda: ops.gemm_relu_gemm(x, *ws, out=out, activation=act, weight_layout=layout))
    assert got == ("few", b * ((M + 127) // 128)) and ops.device_status() == 0
    h = x.double() @ w1.double()
    want = (h.relu() if act == "relu" else h).half().double() @ w2.double()
    _close(out, want, torch.float16)


@pytest.mark.parametrize("a,b,dtype", VALUES)
def test_rows_masked_apart(a, b, dtype):
    g = torch.Generator(device="cuda").manual_seed(14)
    n, M, L, d = 150, 128, 512, 128
    q, k, v = (torch.randn(n, rows, d, generator=g, device="cuda") for rows in (M, L, L))
    v = v.to(dtype)
    q[:, :, 5] = torch.where(torch.arange(M, device="cuda") % 3 == 1, a, 0.0)
    q = q.to(dtype)
    for lo, hi in MASKED:
        kk = k.clone()
        kk[:, :, 5] = 0.0
        kk[:, lo:hi, 5] = b
        kk = kk.to(dtype)
        out = ops.bmm_softmax_bmm(q, kk, v, scale=d ** -0.5, key_layout="LK")
        for i in (0, 75, 149):
            _close(out[i:i + 1], _reference(q[i:i + 1], kk[i:i + 1], v[i:i + 1], d ** -0.5), dtype)
    assert _launched(lambda: ops.bmm_softmax_bmm(q, kk, v, out, scale=d ** -0.5, key_layout="LK")) == ("few", n)
    assert ops.device_status() == 0


@pytest.mark.parametrize("b,M,blocks,act,form", [
    (148, 128, 4, None, "few"), (1000, 128, 2, None, "whole"), (1000, 128, 3, None, "few"), (148, 256, 4, None, "whole"), (74, 512, 4, None, "few"), (148, 256, 8, "relu", "few"),
    (300, 256, 2, "relu", "whole"), (300, 256, 4, "relu", "few"), (100, 512, 4, "relu", "whole")])
def test_form_by_shape(b, M, blocks, act, form):
    q, k, v = _operands(b, M, 128, 128, 128 * blocks, torch.float16, 7)
    out = torch.empty_like(q)
    if act is None:
        got = _launched(lambda: ops.bmm_softmax_bmm(q, k, v, out, scale=0.1, key_layout="LK"))
    else:
        w1 = k.transpose(1, 2).contiguous()
        got = _launched(lambda: ops.gemm_relu_gemm(q, w1, v, out, activation=act))
    assert got[0] == form
