"""Attention and small chains of few items, which take the kernel with two softmax warps per quarter of the rows by themselves, against
float64 products of the same 16-bit operands: every length of a last block, one and several blocks, row tails, widths below
the kernel's, both layouts and types; and, for every form of the attention kernel, single weights and scores that are not finite."""
import ctypes
import re

import pytest
import torch

from ditto_b200 import _lib, ops
from tests.test_gpu_attention_masked_rows import FORMS
from tests.test_gpu_attention_split import _close, _reference

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("N,K", [(64, 64), (16, 48), (128, 128), (80, 80), (112, 16)])
@pytest.mark.parametrize("b,M,L", [(2, 128, 128), (1, 16, 16), (1, 144, 32), (2, 208, 48), (1, 128, 64), (1, 32, 80), (3, 128, 96), (1, 272, 112),
                                   (2, 64, 208), (1, 128, 192), (1, 128, 368)])
def test_shapes(dtype, N, K, b, M, L):
    g = torch.Generator(device="cuda").manual_seed(b * M + L)
    q = torch.randn(b, M, K, generator=g, device="cuda").to(dtype)
    k = torch.randn(b, L, K, generator=g, device="cuda").to(dtype)
    v = torch.randn(b, L, N, generator=g, device="cuda").to(dtype)
    for layout in ("LK", "KL"):
        keys = k if layout == "LK" else k.transpose(1, 2).contiguous()
        out = ops.bmm_softmax_bmm(q, keys, v, scale=2 * K ** -0.5, key_layout=layout)
        assert ops.device_status() == 0
        _close(out, _reference(q, k, v, 2 * K ** -0.5), dtype)
        assert torch.equal(out, ops.bmm_softmax_bmm(q, keys, v, scale=2 * K ** -0.5, key_layout=layout))


@pytest.mark.parametrize("act", ["identity", "relu"])
@pytest.mark.parametrize("layout", ["IO", "OI"])
@pytest.mark.parametrize("b,M,N,K,L", [(1, 144, 64, 64, 80), (2, 16, 128, 96, 208), (3, 128, 16, 64, 512), (74, 128, 64, 64, 1024),
                                       (100, 128, 64, 64, 128), (296, 16, 48, 64, 80)])
def test_chains(act, layout, b, M, N, K, L):
    g = torch.Generator(device="cuda").manual_seed(M + L)
    x = torch.randn(b, M, K, generator=g, device="cuda").half()
    w1 = (torch.randn(b, K, L, generator=g, device="cuda") * K ** -0.5).half()
    w2 = (torch.randn(b, L, N, generator=g, device="cuda") * L ** -0.5).half()
    h = x.double() @ w1.double()
    want = (h.relu() if act == "relu" else h).half().double() @ w2.double()
    ws = (w1, w2) if layout == "IO" else (w1.transpose(1, 2).contiguous(), w2.transpose(1, 2).contiguous())
    out = ops.gemm_relu_gemm(x, *ws, activation=act, weight_layout=layout)
    assert ops.device_status() == 0
    _close(out, want, torch.float16)


def _attention(q, k, v, scale, layout, flags):
    keys = k if layout == "LK" else k.transpose(1, 2).contiguous()
    out = ops.bmm_softmax_bmm(q, keys, v, scale=scale, key_layout=layout, flags=flags)
    assert ops.device_status() == 0
    return out


def _operands(b, M, N, K, L, dtype, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return tuple(torch.randn(b, rows, cols, generator=g, device="cuda").to(dtype) for rows, cols in ((M, K), (L, K), (L, N)))


@pytest.mark.parametrize("code", [0, 2, 3, 4])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("b,M,N,K,L,layout", [
    (3, 128, 64, 64, 1024, "LK"), (2, 208, 64, 64, 1168, "KL"), (1, 16, 64, 64, 256, "LK"), (2, 144, 48, 16, 912, "LK"),
    (3, 128, 128, 128, 1024, "LK"), (2, 272, 80, 80, 1168, "KL"), (1, 16, 16, 128, 272, "LK"), (300, 384, 64, 64, 384, "LK")])
def test_parts(code, dtype, b, M, N, K, L, layout):
    """The kernel by its name, with every number of parts (the last shape: several rounds of CTAs)."""
    q, k, v = _operands(b, M, N, K, L, dtype, b * M + L + code)
    flags = _lib.FLAG_FEW | code * _lib.FLAG_SPLIT_UNIT
    out = _attention(q, k, v, 2 * K ** -0.5, layout, flags)
    _close(out, _reference(q, k, v, 2 * K ** -0.5), dtype)
    assert torch.equal(out, _attention(q, k, v, 2 * K ** -0.5, layout, flags))


FEW, UNIT = _lib.FLAG_FEW, _lib.FLAG_SPLIT_UNIT


class _KernelNode(ctypes.Structure):
    """CUDA_KERNEL_NODE_PARAMS_v2"""
    _fields_ = [("func", ctypes.c_void_p), ("grid", ctypes.c_uint * 3), ("block", ctypes.c_uint * 3), ("shared", ctypes.c_uint),
                ("params", ctypes.c_void_p), ("extra", ctypes.c_void_p), ("kernel", ctypes.c_void_p), ("context", ctypes.c_void_p)]


def _launched(call):
    """The attention kernel that a call launches and its number of CTAs, read from a captured graph."""
    call()
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
        call()
    cuda = ctypes.CDLL("libcuda.so.1")
    handle, count, node, name = ctypes.c_void_p(graph.raw_cuda_graph()), ctypes.c_size_t(1), ctypes.c_void_p(), ctypes.c_char_p()
    params = _KernelNode()
    assert cuda.cuGraphGetNodes(handle, ctypes.byref(node), ctypes.byref(count)) == 0 and count.value == 1
    assert cuda.cuGraphKernelNodeGetParams_v2(node, ctypes.byref(params)) == 0
    if params.func:
        assert cuda.cuFuncGetName(ctypes.byref(name), ctypes.c_void_p(params.func)) == 0
    else:
        assert cuda.cuKernelGetName(ctypes.byref(name), ctypes.c_void_p(params.kernel)) == 0
    kernel, arguments = re.search(r"\d(attention_\w*?kernel)I(\w+?)EEv", name.value.decode()).groups()
    form = {"attention_kernel": "by row" if arguments.endswith("Lb1E") else "whole", "attention_short_kernel": "few",
            "attention_narrow_kernel": "narrow"}.get(kernel, kernel)
    return form, params.grid[0]


@pytest.mark.parametrize("code", [2, 3, 4])
def test_names_lead_to_their_kernels(code):
    q, k, v = _operands(4, 384, 64, 64, 8192, torch.float16, 9)
    out = torch.empty_like(q)
    for flags, name in ((0, "by row"), (FEW, "few")):
        got = _launched(lambda: ops.bmm_softmax_bmm(q, k, v, out, scale=0.125, key_layout="LK", flags=flags | code * UNIT))
        assert got == (name, 12 << (code - 1))


@pytest.mark.parametrize("tiles,blocks,d,act,form,parts", [
    (24, 64, 64, None, "by row", 8), (1, 64, 64, None, "by row", 8), (16, 64, 64, None, "by row", 8),      # many blocks even in eight parts
    (148, 16, 64, None, "by row", 2),          # two CTAs an SM, as many clusters of two as SMs
    (60, 16, 64, None, "few", 4),              # ... clusters of four where a CTA an SM leaves no room for them
    (24, 16, 64, None, "few", 4), (24, 4, 64, None, "few", 4), (24, 2, 64, None, "few", 2), (100, 2, 64, None, "few", 1),
    (296, 3, 64, None, "few", 1), (600, 3, 64, None, "narrow", 1), (1000, 6, 128, None, "few", 1),
    (100, 1, 64, "relu", "few", 1), (296, 1, 64, "identity", "few", 1), (148, 32, 64, "relu", "by row", 2), (24, 8, 64, "identity", "few", 4),
])
def test_form_by_shape(tiles, blocks, d, act, form, parts):
    q, k, v = _operands(tiles, 128, d, d, 128 * blocks, torch.float16, 7)
    out = torch.empty_like(q)
    if act is None:
        got = _launched(lambda: ops.bmm_softmax_bmm(q, k, v, out, scale=d ** -0.5, key_layout="LK"))
    else:
        w1 = k.transpose(1, 2).contiguous()
        got = _launched(lambda: ops.gemm_relu_gemm(q, w1, v, out, activation=act))
    assert got == (form, tiles * parts)


@pytest.mark.parametrize("code", [2, 3])
@pytest.mark.parametrize("b,M,N,K,L,dtype,layout", [(74, 128, 64, 64, 4352, torch.float16, "LK"), (19, 400, 64, 64, 4240, torch.bfloat16, "KL"),
                                                    (37, 256, 48, 32, 4240, torch.float16, "KL"), (9, 144, 64, 64, 8208, torch.bfloat16, "LK")])
def test_long_parts(b, M, N, K, L, dtype, layout, code):
    """Many blocks a part: the split kernel with a thread a row, by its name."""
    q, k, v = _operands(b, M, N, K, L, dtype, b)
    out = _attention(q, k, v, K ** -0.5, layout, code * _lib.FLAG_SPLIT_UNIT)
    for i in range(0, b, 9):
        _close(out[i:i + 1], _reference(q[i:i + 1], k[i:i + 1], v[i:i + 1], K ** -0.5), dtype)


@pytest.mark.parametrize("act", ["identity", "relu"])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("layout", ["IO", "OI"])
@pytest.mark.parametrize("b,M,N,K,L", [(1, 144, 64, 48, 8192), (3, 16, 16, 64, 4176)])
def test_long_chains(b, M, N, K, L, layout, dtype, act):
    """Chains of a few tiles and more than three blocks a part even in eight parts: the split kernel with a thread a row."""
    g = torch.Generator(device="cuda").manual_seed(L)
    x = torch.randn(b, M, K, generator=g, device="cuda").to(dtype)
    w1 = (torch.randn(b, K, L, generator=g, device="cuda") * K ** -0.5).to(dtype)
    w2 = (torch.randn(b, L, N, generator=g, device="cuda") * L ** -0.5).to(dtype)
    h = x.double() @ w1.double()
    want = (h.relu() if act == "relu" else h).to(dtype).double() @ w2.double()
    ws = (w1, w2) if layout == "IO" else (w1.transpose(1, 2).contiguous(), w2.transpose(1, 2).contiguous())
    out = ops.gemm_relu_gemm(x, *ws, activation=act, weight_layout=layout)
    assert ops.device_status() == 0
    _close(out, want, dtype)


@pytest.mark.parametrize("code", [0, 2, 3, 4])
@pytest.mark.parametrize("d", [64, 128])
def test_whole_parts_of_minus_infinity(code, d):
    q, k, v = _operands(1, 128, d, d, 1024, torch.bfloat16, 5)
    q = q.abs() + 0.5
    k[:, 128:] = float("-inf")                       # q is positive: these scores are -inf
    out = _attention(q, k, v, 0.25, "LK", _lib.FLAG_FEW | code * _lib.FLAG_SPLIT_UNIT)
    _close(out, _reference(q, k[:, :128], v[:, :128], 0.25), torch.bfloat16)


@pytest.mark.parametrize("heads,d,M", [(4, 64, 1040), (2, 128, 528)])
def test_packed_heads(heads, d, M):
    g = torch.Generator(device="cuda").manual_seed(M)
    qkv = torch.randn(2, M, 3 * heads * d, generator=g, device="cuda").half()
    q, k, v = (t.reshape(2, M, heads, d).transpose(1, 2).reshape(2 * heads, M, d) for t in qkv.chunk(3, dim=-1))
    want = _reference(q, k, v, d ** -0.5).reshape(2, heads, M, d).transpose(1, 2).reshape(2, M, heads * d)
    for code in (0, 2, 3, 4):
        out = ops.multi_head_attention(qkv, heads, scale=d ** -0.5, flags=_lib.FLAG_FEW | code * _lib.FLAG_SPLIT_UNIT)
        assert ops.device_status() == 0
        _close(out, want, torch.float16)


@pytest.mark.parametrize("b,M,L", [(70, 16, 208), (200, 128, 512), (250, 128, 784), (296, 64, 144), (149, 128, 128)])
@pytest.mark.parametrize("d", [64, 128])
def test_more_items_than_sms(b, M, L, d):
    g = torch.Generator(device="cuda").manual_seed(b)
    q = torch.randn(b, M, d, generator=g, device="cuda").half()
    k = torch.randn(b, L, d, generator=g, device="cuda").half()
    v = torch.randn(b, L, d, generator=g, device="cuda").half()
    for flags in (0, FEW):
        out = _attention(q, k, v, d ** -0.5, "LK", flags)
        for i in range(0, b, 11):
            _close(out[i:i + 1], _reference(q[i:i + 1], k[i:i + 1], v[i:i + 1], d ** -0.5), torch.float16)


ALL_FORMS = {**FORMS, "few items": 0}


@pytest.mark.parametrize("form,d", [(f, d) for f in ALL_FORMS for d in (64, 128) if d == 64 or f != "narrow"])
def test_every_weight(form, d):
    """V is the identity, d keys at a time: the result is the weights themselves.  They differ from float64's by the rounding of
    the 16-bit weight (2^-11, or 2^-25 where it is subnormal: the row's largest is 1 before the division) and of the result."""
    g = torch.Generator(device="cuda").manual_seed(d)
    L = 2 * d + 16
    q = torch.randn(1, 128, d, generator=g, device="cuda").half()
    k = torch.randn(1, L, d, generator=g, device="cuda").half()
    p = torch.softmax(q.double() @ k.double().transpose(1, 2) * 0.5, -1)
    for first in range(0, L, d):
        v = torch.zeros(1, L, d, device="cuda", dtype=torch.float16)
        n = min(d, L - first)
        v[0, first:first + n, :n] = torch.eye(n, device="cuda", dtype=torch.float16)
        out = ops.bmm_softmax_bmm(q, k, v, scale=0.5, key_layout="LK", flags=ALL_FORMS[form])
        want = p[:, :, first:first + n]
        # (a reference up to 2^8 below the maximum makes weights larger and subnormals rarer; the sum's own error is some 2^-13)
        assert ((out[:, :, :n].double() - want).abs() <= 2.0 ** -10 * 1.2 * want + 2.0 ** -24).all()
    assert ops.device_status() == 0


@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
@pytest.mark.parametrize("form,d", [(f, d) for f in ALL_FORMS for d in (64, 128) if d == 64 or f != "narrow"])
def test_rows_with_scores_that_are_not_numbers(form, d, bad):
    """A score of NaN, or of +inf, makes its row NaN as in torch.softmax, wherever the key lies; the other rows are what they were."""
    g = torch.Generator(device="cuda").manual_seed(3)
    q = torch.randn(1, 128, d, generator=g, device="cuda").bfloat16()
    k = torch.randn(1, 400, d, generator=g, device="cuda").bfloat16()
    v = torch.randn(1, 400, d, generator=g, device="cuda").bfloat16()
    q[:, :, 5] = q[:, :, 20] = 0.0
    q[:, 40, 5] = 1e30                                # the product overflows float32 in that row alone
    for key in (0, 7, 100, 127, 128, 250, 391, 399):
        kk = k.clone()
        kk[:, :, 5] = 0.0
        kk[:, key, 5] = 1e30
        qq = q.clone()
        if bad != bad:
            qq[:, 40, 20], kk[:, key, 20] = 1e30, -1e30   # inf - inf
        out = ops.bmm_softmax_bmm(qq, kk, v, scale=0.125, key_layout="LK", flags=ALL_FORMS[form])
        assert out[:, 40].isnan().all()
        keep = [i for i in range(128) if i != 40]
        _close(out[:, keep], _reference(qq[:, keep], kk, v, 0.125), torch.bfloat16)
    assert ops.device_status() == 0


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("b,L", [(24, 208), (128, 512), (32, 512)])
def test_no_less_precise_than_the_other_kernels(b, L, dtype):
    """The norm of the error against float64 beside those of the 64-key kernel and of the one with a thread a row.  The error is the
    rounding of some 10^5 results and more, so that two kernels of the same precision differ by about 1 %."""
    g = torch.Generator(device="cuda").manual_seed(L)
    q = torch.randn(b, 256, 64, generator=g, device="cuda").to(dtype)
    k = torch.randn(b, L, 64, generator=g, device="cuda").to(dtype)
    v = torch.randn(b, L, 64, generator=g, device="cuda").to(dtype)
    for scale in (0.125, 0.35, 1.0):
        want = _reference(q, k, v, scale)
        few, narrow, whole = ((ops.bmm_softmax_bmm(q, k, v, scale=scale, key_layout="LK", flags=f).double() - want).norm().item()
                              for f in (FEW, _lib.FLAG_NARROW, UNIT))
        assert few <= 1.01 * max(narrow, whole), (scale, few, narrow, whole)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("b,L,code", [(6, 6096, 4), (13, 7056, 3), (37, 2304, 2)])
def test_long_parts_no_less_precise_than_short_ones(b, L, code, dtype):
    """The two kernels whose parts a call may get, split alike, on operands whose scores spread (U(-1, 1), unscaled): the norms of their
    errors against float64 over 5 * 10^4 results and more differ by about 1 %."""
    g = torch.Generator(device="cuda").manual_seed(L)
    q, k, v = ((2 * torch.rand(b, rows, 64, generator=g, device="cuda") - 1).to(dtype) for rows in (128, L, L))
    want = _reference(q, k, v, 1.0)
    by_row, few = ((_attention(q, k, v, 1.0, "LK", f | code * UNIT).double() - want).norm().item() for f in (0, FEW))
    assert by_row <= 1.01 * few, (by_row, few)
