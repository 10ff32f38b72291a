"""Where calls go over from one form of attention and of small chains to another at two to nine items an SM: the kernel, its CTAs and the shared memory they ask
for, read from a captured graph, on either side of each line; and that the results of either side are those of float64 products."""
import ctypes

import pytest
import torch

from ditto_b200 import ops
from tests.test_gpu_attention_short import _KernelNode, _launched, _operands
from tests.test_gpu_attention_split import _close, _reference

pytestmark = pytest.mark.gpu


def _case(b, M, N, K, L, act, dtype=torch.float16):
    """A call into a result of its own, that result, and the float64 products of some of its slices."""
    q, k, v = _operands(b, M, N, K, L, dtype, b + M + L)
    out = torch.full((b, M, N), float("nan"), dtype=dtype, device="cuda")
    if act is None:
        return (lambda: ops.bmm_softmax_bmm(q, k, v, out, scale=K ** -0.5, key_layout="LK")), out, \
            lambda i: _reference(q[i:i + 1], k[i:i + 1], v[i:i + 1], K ** -0.5)
    k, v = (k.float() * K ** -0.5).to(dtype), (v.float() * L ** -0.5).to(dtype)
    w1 = k.transpose(1, 2).contiguous()

    def want(i):
        h = q[i:i + 1].float() @ w1[i:i + 1].float()
        return ((h.relu() if act == "relu" else h).to(dtype).float() @ v[i:i + 1].float()).double()
    return (lambda: ops.gemm_relu_gemm(q, w1, v, out=out, activation=act)), out, want


def _check(call, out, want):
    call()
    assert ops.device_status() == 0
    for i in range(0, out.shape[0], 97):
        _close(out[i:i + 1], want(i), out.dtype)


# one tile a sequence: two CTAs an SM (few), or the kernel that asks for an item's operands under the one before (whole)
@pytest.mark.parametrize("b,M,N,K,L,act,form", [
    (296, 128, 128, 128, 128, "identity", "few"), (297, 128, 128, 128, 128, "identity", "whole"), (444, 128, 80, 80, 64, "relu", "whole"),      # chains of one block
    (444, 48, 128, 128, 96, "identity", "few"), (297, 64, 128, 128, 96, "identity", "whole"), (297, 48, 128, 128, 112, "relu", "whole"),
    (400, 128, 128, 128, 256, "identity", "few"), (401, 128, 128, 128, 256, "identity", "whole"), (444, 80, 128, 128, 256, "identity", "few"),
    (444, 128, 96, 96, 256, "identity", "few"), (445, 128, 96, 96, 256, "identity", "whole"),
    (380, 128, 128, 128, 128, None, "few"), (381, 128, 128, 128, 128, None, "whole"), (444, 80, 128, 128, 128, None, "few"), (445, 80, 128, 128, 128, None, "whole"),
    (425, 112, 112, 112, 96, None, "few"), (426, 112, 112, 112, 96, None, "whole"), (444, 128, 64, 128, 128, None, "few"), (444, 128, 128, 128, 64, None, "few"),
    (444, 112, 128, 128, 160, None, "few"), (445, 112, 128, 128, 160, None, "whole"),
    (2000, 128, 128, 128, 384, None, "few"), (2000, 128, 128, 128, 384, "identity", "few")])
def test_one_tile_a_sequence(b, M, N, K, L, act, form):
    call, out, want = _case(b, M, N, K, L, act)
    _check(call, out, want)
    assert _launched(call)[0] == form


# chains of two tiles a sequence
@pytest.mark.parametrize("b,N,K,L,form", [
    (518, 128, 128, 512, "few"), (519, 128, 128, 512, "whole"), (519, 128, 128, 1040, "few"), (519, 128, 128, 1024, "whole"), (666, 96, 96, 512, "few"),
    (667, 96, 96, 512, "whole"), (667, 80, 80, 1024, "few"), (667, 64, 128, 912, "few"), (667, 64, 128, 896, "whole"), (300, 128, 128, 384, "whole")])
def test_chains_of_two_tiles_a_sequence(b, N, K, L, form):
    call, out, want = _case(b, 208, N, K, L, "relu")
    _check(call, out, want)
    assert _launched(call)[0] == form


def _shared(call):
    """Kernel, CTAs and shared memory of the one launch of a call."""
    form, ctas = _launched(call)
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
        call()
    cuda, count, node, params = ctypes.CDLL("libcuda.so.1"), ctypes.c_size_t(1), ctypes.c_void_p(), _KernelNode()
    assert cuda.cuGraphGetNodes(ctypes.c_void_p(graph.raw_cuda_graph()), ctypes.byref(node), ctypes.byref(count)) == 0
    assert cuda.cuGraphKernelNodeGetParams_v2(node, ctypes.byref(params)) == 0
    return form, ctas, params.shared


# head dimension 64, three items an SM at most: places for three CTAs an SM, or for four where one block of 64 keys is the whole item
@pytest.mark.parametrize("b,L,act,places", [
    (444, 80, "identity", 3), (445, 80, "identity", 4), (370, 64, "identity", 3), (371, 64, "identity", 4), (444, 16, "relu", 4), (425, 64, None, 3),
    (426, 64, None, 4), (444, 80, None, 3), (297, 64, None, 3), (297, 16, "identity", 3)])
def test_places_of_the_kernel_with_64_key_blocks(b, L, act, places):
    call, out, want = _case(b, 128, 64, 64, L, act)
    _check(call, out, want)
    form, ctas, shared = _shared(call)
    assert form == "narrow" and ctas == b and (228 << 10) // (shared + 1024) == places
