"""Calls of two to three items an SM at head dimensions up to 64: the kernel with 64-key blocks with places for three CTAs an SM, for any number
of blocks, against float64 products, one call after another; and the sizes at which the rule hands over."""
import pytest
import torch

from ditto_b200 import ops
from tests.test_gpu_attention_short import _launched
from tests.test_gpu_attention_split import _close, _reference

pytestmark = pytest.mark.gpu


def _operands(b, M, N, K, L, dtype):
    g = torch.Generator(device="cuda").manual_seed(b + M + L)
    return [torch.randn(b, *size, device="cuda", generator=g).to(dtype) for size in ((M, K), (L, K), (L, N))]


# items on either side of the lines, one block and many, a partial last block, row tails
@pytest.mark.parametrize("b,M,N,K,L,act,form", [
    (297, 128, 64, 64, 1040, None, "narrow"), (444, 16, 64, 64, 48, None, "narrow"), (148, 272, 48, 32, 2192, None, "narrow"), (99, 400, 64, 64, 8192, None, "narrow"),
    (297, 128, 64, 64, 640, "relu", "narrow"), (148, 384, 16, 64, 2192, "identity", "narrow"), (296, 128, 64, 64, 1040, None, "other"),
    (445, 128, 64, 64, 3088, None, "other"), (445, 128, 64, 64, 3072, None, "narrow"), (445, 128, 64, 64, 400, "relu", "other"), (445, 128, 64, 64, 256, "relu", "narrow")])
@pytest.mark.parametrize("dtype,layout", [(torch.float16, "LK"), (torch.bfloat16, "KL")])
def test_calls_one_after_another(b, M, N, K, L, act, form, dtype, layout):
    q, k, v = _operands(b, M, N, K, L, dtype)
    outs = [torch.full((b, M, N), float("nan"), dtype=dtype, device="cuda") for _ in range(3)]
    if act is None:
        keys = k if layout == "LK" else k.transpose(1, 2).contiguous()
        call = lambda out: ops.bmm_softmax_bmm(q, keys, v, out, scale=K ** -0.5, key_layout=layout)
        want = lambda i: _reference(q[i:i + 1], k[i:i + 1], v[i:i + 1], K ** -0.5)
    else:
        k = (k.float() * K ** -0.5).to(dtype)
        v = (v.float() * L ** -0.5).to(dtype)
        ws = (k.transpose(1, 2).contiguous(), v) if layout == "KL" else (k, v.transpose(1, 2).contiguous())
        call = lambda out: ops.gemm_relu_gemm(q, *ws, out, activation=act, weight_layout="IO" if layout == "KL" else "OI")

        def want(i):
            h = q[i:i + 1].float() @ k[i:i + 1].float().transpose(1, 2)
            return ((h.relu() if act == "relu" else h).to(dtype).float() @ v[i:i + 1].float()).double()
    for out in outs:
        call(out)
    assert ops.device_status() == 0
    for i in range(0, b, 37):
        _close(outs[0][i:i + 1], want(i), dtype)
    assert torch.equal(outs[0], outs[1]) and torch.equal(outs[0], outs[2])
    got, ctas = _launched(lambda: call(outs[0]))
    assert (got == "narrow") == (form == "narrow") and (got != "narrow" or ctas == b * ((M + 127) // 128))
