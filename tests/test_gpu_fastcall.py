"""The native call path against the checked Python path: the same calls give the same bits and shapes, and what the checked
path refuses is refused with its errors, whichever path saw the call first."""
import pytest
import torch

from ditto_b200 import ops

pytestmark = pytest.mark.gpu


def _both(fn):
    """Results (or error types) of the native and of the checked path."""
    got = []
    fast = ops._fast
    for path in (fast, None):
        ops._fast = path
        try:
            got.append(fn())
        except Exception as e:                          # noqa: BLE001 - the error is the result
            got.append((type(e), str(e)))
        finally:
            ops._fast = fast
    return got


def _t(*shape, dtype=torch.float16, device="cuda"):
    return torch.randn(*shape, device=device).to(dtype)


def _calls():
    q, k, v = _t(2, 144, 64), _t(2, 272, 64), _t(2, 272, 48)
    x, w1, w2 = _t(48, 128), _t(128, 320), _t(320, 256)
    qkv = _t(2, 64, 3 * 128)
    yield "softmax", lambda: ops.bmm_softmax_bmm(q, k, v, scale=0.125, key_layout="LK")
    yield "integer scale and flags", lambda: ops.bmm_softmax_bmm(q, k, v, scale=1, key_layout="LK", flags=2)
    yield "given result", lambda: ops.bmm_softmax_bmm(q, k, v, out=torch.empty(2, 144, 48, device="cuda", dtype=q.dtype),
                                                      scale=0.125, key_layout="LK")
    yield "heads", lambda: ops.multi_head_attention(qkv, 2, scale=0.5)
    yield "chain", lambda: ops.gemm_relu_gemm(x, w1, w2)
    yield "batched chain", lambda: ops.gemm_relu_gemm(x[None], w1[None], w2[None], activation="identity")
    yield "flat result of a batch of one", lambda: ops.gemm_relu_gemm(x[None], w1[None], w2[None],
                                                                      out=torch.empty(48, 256, device="cuda", dtype=x.dtype))
    yield "no scratch", lambda: ops.gemm_relu_gemm(x, w1, w2, workspace=None)
    yield "ffn", lambda: ops.ffn(x, w1, _t(320) * 0 + 1, w2, None, act1="gelu", act2="identity", weight_layout="IO")
    yield "requires grad", lambda: ops.gemm_relu_gemm(x.clone().requires_grad_(), w1, w2)
    # refused
    yield "wrong key layout", lambda: ops.bmm_softmax_bmm(q, k, v, key_layout="KL")
    yield "unknown layout", lambda: ops.bmm_softmax_bmm(q, k, v, key_layout="XX")
    yield "float32", lambda: ops.bmm_softmax_bmm(q.float(), k.float(), v.float(), key_layout="LK")
    yield "mixed types", lambda: ops.bmm_softmax_bmm(q, k.bfloat16(), v, key_layout="LK")
    yield "host tensor", lambda: ops.bmm_softmax_bmm(q.cpu(), k, v, key_layout="LK")
    yield "not a tensor", lambda: ops.bmm_softmax_bmm([1], k, v, key_layout="LK")
    yield "strided", lambda: ops.bmm_softmax_bmm(q.transpose(0, 1), k, v, key_layout="LK")
    yield "wrong result shape", lambda: ops.bmm_softmax_bmm(q, k, v, out=torch.empty_like(q), key_layout="LK")
    yield "text scale", lambda: ops.bmm_softmax_bmm(q, k, v, scale="x", key_layout="LK")
    yield "negative scale", lambda: ops.bmm_softmax_bmm(q, k, v, scale=-1.0, key_layout="LK")
    yield "rows not of 16", lambda: ops.bmm_softmax_bmm(q[:, :100].contiguous(), k, v, key_layout="LK")
    yield "misaligned", lambda: ops.gemm_relu_gemm(_t(48 * 128 + 1)[1:].view(48, 128), w1, w2)
    yield "empty", lambda: ops.gemm_relu_gemm(x[:0], w1, w2)
    yield "heads that do not divide", lambda: ops.multi_head_attention(qkv, 5)
    yield "no heads", lambda: ops.multi_head_attention(qkv, 0)
    yield "unknown activation", lambda: ops.gemm_relu_gemm(x, w1, w2, activation="gelu")
    yield "short bias", lambda: ops.ffn(x, w1, _t(319), w2, None, weight_layout="IO")


def test_native_path_answers_like_the_checked_path(cuda):
    ops.bmm_softmax_bmm(_t(1, 16, 16), _t(1, 16, 16), _t(1, 16, 16), key_layout="LK")     # sets the native path up
    assert ops._fast is not None
    torch.manual_seed(3)
    for name, call in _calls():
        native, checked = _both(call)
        if isinstance(checked, tuple):
            assert native == checked, name
        else:
            assert native.shape == checked.shape and native.dtype == checked.dtype and torch.equal(native, checked), name
    assert ops.device_status(cuda) == 0
