"""Which kernels calls of the MLP chain with scratch memory take, by the names in a captured graph -- the size of the scratch memory does not tell,
since the wave kernel asks for what the tile or the flow kernel would -- and those kernels' results where calls of the same sizes else take the wave
kernel: every cut of the tile kernel and every epilogue of the flow kernel, reached by results that are aligned to 16 bytes alone."""
import ctypes
import re

import pytest
import torch

from ditto_b200 import _lib, ops
from tests import test_gpu_mlp_flow as flow
from tests import test_gpu_mlp_tiles as tiles
from tests.test_gpu_attention_short import _KernelNode
from tests.test_gpu_random_shapes import _act, _assert_close

pytestmark = pytest.mark.gpu

TILES, WAVES, FLOW = ["mlp_tiles_kernel"] * 2, ["mlp_waves_kernel"] * 2, ["mlp_flow_reset_kernel", "mlp_flow_kernel"]


def _kernels(call, sizes=None):
    """The kernels that a call launches, in order of launch (and in `sizes` how many kernels the module of each holds)."""
    call()
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
        call()
    cuda, names, module, held = ctypes.CDLL("libcuda.so.1"), [], ctypes.c_void_p(), ctypes.c_uint(0)
    handle, count = ctypes.c_void_p(graph.raw_cuda_graph()), ctypes.c_size_t(0)
    assert cuda.cuGraphGetNodes(handle, None, ctypes.byref(count)) == 0
    nodes = (ctypes.c_void_p * count.value)()
    assert cuda.cuGraphGetNodes(handle, nodes, ctypes.byref(count)) == 0
    for node in nodes:
        params, name = _KernelNode(), ctypes.c_char_p()
        assert cuda.cuGraphKernelNodeGetParams_v2(ctypes.c_void_p(node), ctypes.byref(params)) == 0
        if params.func:
            assert cuda.cuFuncGetName(ctypes.byref(name), ctypes.c_void_p(params.func)) == 0
            if sizes is not None:
                assert cuda.cuFuncGetModule(ctypes.byref(module), ctypes.c_void_p(params.func)) == 0
                assert cuda.cuModuleGetFunctionCount(ctypes.byref(held), module) == 0
        else:
            assert cuda.cuKernelGetName(ctypes.byref(name), ctypes.c_void_p(params.kernel)) == 0
            if sizes is not None:
                assert cuda.cuKernelGetLibrary(ctypes.byref(module), ctypes.c_void_p(params.kernel)) == 0
                assert cuda.cuLibraryGetKernelCount(ctypes.byref(held), module) == 0
        if sizes is not None:
            sizes.append(held.value)
        names.append(re.search(r"\d(mlp_\w*?kernel)", name.value.decode()).group(1))
    return names


def _half_aligned(cuda, batch, M, N, dtype):
    """A result at an address that is a multiple of 16 and not of 32."""
    out = torch.full((batch * M * N + 16,), float("nan"), dtype=dtype, device=cuda)[8:8 + batch * M * N].view(batch, M, N)
    assert out.data_ptr() % 32 == 16
    return out


# biases at addresses that allow 16-byte loads and at such that do not, and one bias missing
def _biases(cuda, g, batch, N, L, dtype):
    bias = (torch.randn(batch * (L + N) + 2, device=cuda, generator=g) * 0.5).to(dtype)
    return ((bias[:batch * L], bias[batch * L:batch * (L + N)]), (bias[2:2 + batch * L], None), (None, bias[2:2 + batch * N]))


def _check_ffn(cuda, shape, x, w1, w2, given, b1, b2, act1, act2, layout, out):
    batch, M, N, K, L = shape
    ops.ffn(x, given[0], b1, given[1], b2, out=out, act1=act1, act2=act2, weight_layout=layout)
    h = x.float() @ w1.float() + (0 if b1 is None else b1.float().view(batch, 1, L))
    y = _act(h, act1).to(x.dtype).float() @ w2.float() + (0 if b2 is None else b2.float().view(batch, 1, N))
    _assert_close(out, _act(y, act2), x.dtype, ("ffn", act1, act2, b1 is None, b2 is None, layout) + shape, cuda)


@pytest.mark.parametrize("shape", tiles.SHAPES)
@pytest.mark.parametrize("layout", ["IO", "OI"])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_every_cut_in_the_tile_kernel(cuda, shape, layout, dtype):
    batch, M, N, K, L = shape
    g, x, w1, w2 = tiles._operands(cuda, *shape, dtype, 61)
    given = (w1, w2) if layout == "IO" else (w1.transpose(1, 2).contiguous(), w2.transpose(1, 2).contiguous())
    out = _half_aligned(cuda, batch, M, N, dtype)
    call = lambda: ops.gemm_relu_gemm(x, *given, out=out, weight_layout=layout)     # noqa: E731
    assert _kernels(call) == TILES
    out.fill_(float("nan"))
    call()
    _assert_close(out, torch.relu(x.float() @ w1.float()).to(dtype).float() @ w2.float(), dtype, ("chain",) + shape, cuda)
    for b1, b2 in _biases(cuda, g, batch, N, L, dtype):
        assert _kernels(lambda: ops.ffn(x, given[0], b1, given[1], b2, out=out, act1="gelu", act2="relu", weight_layout=layout)) == TILES
        out.fill_(float("nan"))
        _check_ffn(cuda, shape, x, w1, w2, given, b1, b2, "gelu", "relu", layout, out)


@pytest.mark.parametrize("shape", flow.LARGE + ((1, 24592, 256, 144, 1024), (3, 8208, 256, 208, 1024)))
@pytest.mark.parametrize("layout", ["IO", "OI"])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_every_epilogue_in_the_flow_kernel(cuda, shape, layout, dtype):
    """(the last two: from two k-steps on the wave kernel takes the call unless its result is not aligned)"""
    batch, M, N, K, L = shape
    g, x, w1, w2, given = flow._operands(cuda, *shape, dtype, layout, 62)
    out = _half_aligned(cuda, batch, M, N, dtype)
    for acts in (("relu", "relu"), ("gelu", "identity"), ("relu", "identity"), ("gelu", "relu"), ("identity", "gelu")):
        for b1, b2 in _biases(cuda, g, batch, N, L, dtype):
            out.fill_(float("nan"))
            _check_ffn(cuda, shape, x, w1, w2, given, b1, b2, *acts, layout, out)
    call = lambda y: ops.ffn(x, given[0], b1, given[1], b2, out=y, act1="gelu", weight_layout=layout)     # noqa: E731
    assert _kernels(lambda: call(out)) == FLOW
    assert _kernels(lambda: call(torch.empty_like(out, memory_format=torch.contiguous_format))) == (FLOW if K < 128 else WAVES)


@pytest.mark.parametrize("shape,kernels", [
    ((64, 128, 1024, 512, 4096), ["mlp_wide_kernel"]), ((33, 336, 1024, 256, 4096), ["mlp_wide_kernel"]), ((40, 128, 1024, 1024, 4096), TILES),
    ((60, 112, 1280, 256, 5120), TILES), ((520, 128, 256, 64, 1024), TILES), ((400, 128, 512, 64, 2048), ["mlp_wide_kernel"]),
    ((24, 384, 768, 768, 3072), WAVES), ((16, 512, 1024, 1024, 4096), WAVES), ((1, 2064, 1024, 1024, 4096), WAVES), ((1, 4096, 768, 768, 3072), WAVES),
    ((1, 512, 768, 768, 3072), TILES)])
def test_form_by_shape(cuda, shape, kernels):
    _, x, w1, w2 = tiles._operands(cuda, *shape, torch.bfloat16, 63)
    out = torch.empty(shape[:3], dtype=torch.bfloat16, device=cuda)
    assert _kernels(lambda: ops.gemm_relu_gemm(x, w1, w2, out=out))[-len(kernels):] == kernels


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_a_workspace_with_room_for_the_ring_alone(cuda, dtype):
    """A call that names no kernel and would keep its whole hidden layer takes the flow kernel, with the same bits."""
    shape = (1, 65552, 256, 128, 1024)
    _, x, w1, w2 = tiles._operands(cuda, *shape, dtype, 64)
    need = _lib.load().ditto_b200_workspace_bytes
    ring, full = (need(_lib.OP_GEMM_RELU_GEMM | bits, *shape, _lib.DTYPE_BF16) for bits in (_lib.EPILOGUE_FLOW_MMA, 0))
    out = torch.empty(shape[:3], dtype=dtype, device=cuda)
    got = []
    for size, kernels in ((full, WAVES), (full - 16, FLOW), (ring, FLOW)):
        ws = torch.full((size,), 0xA5, dtype=torch.uint8, device=cuda)
        assert _kernels(lambda: ops.gemm_relu_gemm(x, w1, w2, out=out, workspace=ws)) == kernels
        got.append(ops.gemm_relu_gemm(x, w1, w2, workspace=ws))
    assert torch.equal(got[0], got[1]) and torch.equal(got[0], got[2])
    _assert_close(got[2], torch.relu(x.float() @ w1.float()).to(dtype).float() @ w2.float(), dtype, shape, cuda)


@pytest.mark.parametrize("shape,kernels,most", [((1, 4096, 768, 768, 3072), WAVES, 9), ((1, 512, 768, 768, 3072), TILES, 60)])
def test_a_first_call_loads_no_more_than_its_form(cuda, shape, kernels, most):
    """A program's first call loads the module of its kernels: the instances are compiled by type, layout and bias, a module each."""
    _, x, w1, w2 = tiles._operands(cuda, *shape, torch.bfloat16, 65)
    out = torch.empty(shape[:3], dtype=torch.bfloat16, device=cuda)
    sizes = []
    assert _kernels(lambda: ops.gemm_relu_gemm(x, w1, w2, out=out), sizes) == kernels
    assert len(sizes) == 2 and max(sizes) <= most, sizes
