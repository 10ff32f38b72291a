"""The attention kernel with an item's keys divided between the CTAs of a cluster, against float32 products of the same
16-bit operands: every number of parts, uneven and minimal parts, partial last blocks, row tails, widths below the
kernel's, both key layouts and types, the chains without a softmax, and scores of -inf filling whole parts."""
import pytest
import torch

from ditto_b200 import _lib, ops

pytestmark = pytest.mark.gpu


def _reference(q, k, v, scale):
    s = (q.double() @ k.double().transpose(1, 2)) * scale
    return torch.softmax(s, -1) @ v.double()


def _close(got, want, dtype):
    # P and the result are rounded once each to the 16-bit type (unit roundoff 2^-11 / 2^-8); P's errors average out
    # over the keys, and |out| <= max |v| bounds them where they do not
    u = 2.0 ** -11 if dtype == torch.float16 else 2.0 ** -8
    err = (got.double() - want).abs()
    assert torch.isfinite(got).all()
    assert (err <= 4 * u * want.abs() + 4 * u * want.pow(2).mean().sqrt()).all(), float(err.max())


@pytest.mark.parametrize("code", [1, 2, 3, 4])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("b,M,N,K,L,layout", [
    (3, 128, 64, 64, 1024, "LK"),      # equal parts
    (2, 208, 64, 64, 1168, "KL"),      # ten blocks, the last of 16 keys, a row tail
    (1, 16, 64, 64, 256, "LK"),        # one row group, one block a part
    (2, 144, 48, 16, 912, "LK"),       # widths below the kernel's
    (3, 128, 128, 128, 1024, "LK"),
    (2, 272, 80, 80, 1168, "KL"),
    (1, 16, 16, 128, 272, "LK"),       # one stored piece: some CTAs of the cluster write nothing
    (40, 384, 64, 64, 384, "LK"),      # more clusters than the device holds at once
])
def test_parts(code, dtype, b, M, N, K, L, layout):
    g = torch.Generator(device="cuda").manual_seed(b * M + L + code)
    q = torch.randn(b, M, K, generator=g, device="cuda").to(dtype)
    k = torch.randn(b, L, K, generator=g, device="cuda").to(dtype)
    v = torch.randn(b, L, N, generator=g, device="cuda").to(dtype)
    keys = k if layout == "LK" else k.transpose(1, 2).contiguous()
    out = ops.bmm_softmax_bmm(q, keys, v, scale=2 * K ** -0.5, key_layout=layout, flags=code * _lib.FLAG_SPLIT_UNIT)
    assert ops.device_status() == 0
    _close(out, _reference(q, k, v, 2 * K ** -0.5), dtype)
    again = ops.bmm_softmax_bmm(q, keys, v, scale=2 * K ** -0.5, key_layout=layout, flags=code * _lib.FLAG_SPLIT_UNIT)
    assert torch.equal(out, again)


@pytest.mark.parametrize("code", [0, 2, 3, 4])
@pytest.mark.parametrize("d", [64, 128])
def test_whole_parts_of_minus_infinity(code, d):
    """Rows whose scores are -inf in all blocks but the first: parts without one finite score contribute nothing."""
    dtype = torch.bfloat16
    g = torch.Generator(device="cuda").manual_seed(5)
    b, M, L = 1, 128, 1024
    q = torch.rand(b, M, d, generator=g, device="cuda").to(dtype) + 0.5
    k = torch.randn(b, L, d, generator=g, device="cuda").to(dtype)
    k[:, 128:] = float("-inf")                       # q is positive: these scores are -inf
    v = torch.randn(b, L, d, generator=g, device="cuda").to(dtype)
    out = ops.bmm_softmax_bmm(q, k, v, scale=0.25, key_layout="LK", flags=code * _lib.FLAG_SPLIT_UNIT)
    assert ops.device_status() == 0
    _close(out, _reference(q[:, :], k[:, :128], v[:, :128], 0.25), dtype)


@pytest.mark.parametrize("act", ["identity", "relu"])
@pytest.mark.parametrize("layout", ["IO", "OI"])
@pytest.mark.parametrize("b,M,N,K,L", [(1, 144, 64, 64, 1168), (2, 16, 128, 96, 2048), (1, 128, 16, 64, 4096)])
def test_chains(act, layout, b, M, N, K, L):
    g = torch.Generator(device="cuda").manual_seed(M + L)
    x = torch.randn(b, M, K, generator=g, device="cuda").half()
    w1 = (torch.randn(b, K, L, generator=g, device="cuda") * K ** -0.5).half()
    w2 = (torch.randn(b, L, N, generator=g, device="cuda") * L ** -0.5).half()
    h = x.double() @ w1.double()
    want = (h.relu() if act == "relu" else h) @ w2.double()
    ws = (w1, w2) if layout == "IO" else (w1.transpose(1, 2).contiguous(), w2.transpose(1, 2).contiguous())
    out = ops.gemm_relu_gemm(x, *ws, activation=act, weight_layout=layout)
    assert ops.device_status() == 0
    _close(out, want, torch.float16)


@pytest.mark.parametrize("heads,d,M", [(4, 64, 1040), (2, 128, 528)])
def test_packed_heads(heads, d, M):
    g = torch.Generator(device="cuda").manual_seed(M)
    qkv = torch.randn(1, M, 3 * heads * d, generator=g, device="cuda").half()
    q, k, v = (t.reshape(M, heads, d).transpose(0, 1) for t in qkv[0].chunk(3, dim=-1))
    want = _reference(q, k, v, d ** -0.5).transpose(0, 1).reshape(1, M, heads * d)
    for code in (0, 2, 3, 4):
        out = ops.multi_head_attention(qkv, heads, scale=d ** -0.5, flags=code * _lib.FLAG_SPLIT_UNIT)
        assert ops.device_status() == 0
        _close(out, want, torch.float16)
