"""The wave kernel, which larger calls of the MLP chain with scratch memory take, at the sizes where it can go wrong, against float32
products (bounds as in the random-shape sweeps): all three tile widths for either GEMM, partial row blocks, tiles past the
hidden layer, odd and half-filled k-steps, several rounds of tiles, batch entries; and what the rule on sizes and alignment picks."""
import ctypes
import re

import pytest
import torch

from ditto_b200 import ops
from tests.test_gpu_attention_short import _KernelNode
from tests.test_gpu_random_shapes import _act, _assert_close

pytestmark = pytest.mark.gpu

# batch, M, N, K, L -> tile widths of the two GEMMs: every pair of widths, even and odd numbers of k-steps
SHAPES = (((1, 8992, 256, 288, 192), (128, 128)), ((1, 7984, 256, 480, 192), (128, 128)), ((1, 7712, 1280, 144, 64), (128, 192)),
          ((1, 4816, 2048, 608, 64), (128, 192)), ((1, 6224, 2048, 144, 64), (128, 256)), ((3, 2928, 256, 208, 320), (192, 128)),
          ((1, 8400, 256, 144, 384), (192, 128)), ((1, 5104, 512, 304, 512), (192, 192)), ((1, 8800, 512, 208, 320), (192, 256)),
          ((1, 4080, 512, 224, 896), (256, 128)), ((1, 8528, 256, 592, 448), (256, 128)), ((3, 2016, 256, 272, 640), (256, 128)),
          ((1, 2064, 1024, 1024, 4096), (256, 128)), ((1, 5280, 512, 416, 640), (256, 192)), ((1, 4096, 768, 768, 3072), (256, 192)),
          ((3, 1312, 1024, 1136, 576), (192, 256)), ((1, 8096, 512, 368, 448), (256, 256)), ((1, 3344, 1280, 1280, 5120), (256, 256)),
          ((24, 384, 768, 768, 3072), (256, 256)))


def _widths(call):
    """Tile widths of a call's two launches if they are the wave kernel's, else its kernels' names, read from a captured graph."""
    call()
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
        call()
    cuda = ctypes.CDLL("libcuda.so.1")
    handle, count = ctypes.c_void_p(graph.raw_cuda_graph()), ctypes.c_size_t(2)
    nodes, names = (ctypes.c_void_p * 2)(), []
    assert cuda.cuGraphGetNodes(handle, nodes, ctypes.byref(count)) == 0 and count.value == 2
    for node in nodes:
        params, name = _KernelNode(), ctypes.c_char_p()
        assert cuda.cuGraphKernelNodeGetParams_v2(ctypes.c_void_p(node), ctypes.byref(params)) == 0
        if params.func:
            assert cuda.cuFuncGetName(ctypes.byref(name), ctypes.c_void_p(params.func)) == 0
        else:
            assert cuda.cuKernelGetName(ctypes.byref(name), ctypes.c_void_p(params.kernel)) == 0
        m = re.search(r"mlp_waves_kernelILb[01]ELi\dELb[01]ELi(\d+)", name.value.decode())
        names.append(int(m.group(1)) if m else re.search(r"\d(mlp_\w*?kernel)", name.value.decode()).group(1))
    return tuple(names)


def _operands(cuda, batch, M, N, K, L, dtype, layout, seed):
    g = torch.Generator(device=cuda).manual_seed(seed)
    x = torch.randn(batch, M, K, device=cuda, generator=g).to(dtype)
    w1 = (torch.randn(batch, K, L, device=cuda, generator=g) * K ** -0.5).to(dtype)
    w2 = (torch.randn(batch, L, N, device=cuda, generator=g) * L ** -0.5).to(dtype)
    given = (w1, w2) if layout == "IO" else (w1.transpose(1, 2).contiguous(), w2.transpose(1, 2).contiguous())
    return g, x, w1, w2, given


@pytest.mark.parametrize("shape,widths", SHAPES)
@pytest.mark.parametrize("layout", ["IO", "OI"])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_wave_kernel(cuda, shape, widths, layout, dtype):
    batch, M, N, K, L = shape
    g, x, w1, w2, given = _operands(cuda, *shape, dtype, layout, 51)
    for act in ("relu", "identity"):
        out = torch.full((batch, M, N), float("nan"), dtype=dtype, device=cuda)
        ops.gemm_relu_gemm(x, *given, out=out, activation=act, weight_layout=layout)
        ref = _act(x.float() @ w1.float(), act).to(dtype).float() @ w2.float()
        _assert_close(out, ref, dtype, (act,) + shape, cuda)
        assert torch.equal(out, ops.gemm_relu_gemm(x, *given, activation=act, weight_layout=layout))
    assert _widths(lambda: ops.gemm_relu_gemm(x, *given, out=out, weight_layout=layout)) == widths
    # biases at addresses that allow 16-byte loads and at such that do not, and one bias missing
    bias = (torch.randn(batch * (L + N) + 2, device=cuda, generator=g) * 0.5).to(dtype)
    for b1, b2, act1, act2 in ((bias[:batch * L], bias[batch * L:batch * (L + N)], "gelu", "identity"), (bias[2:2 + batch * L], None, "gelu", "relu"),
                               (None, bias[2:2 + batch * N], "relu", "gelu")):
        out = ops.ffn(x, given[0], b1, given[1], b2, act1=act1, act2=act2, weight_layout=layout)
        h = x.float() @ w1.float() + (0 if b1 is None else b1.float().view(batch, 1, L))
        y = _act(h, act1).to(dtype).float() @ w2.float() + (0 if b2 is None else b2.float().view(batch, 1, N))
        _assert_close(out, _act(y, act2), dtype, (act1, act2) + shape, cuda)


@pytest.mark.parametrize("shape,form", [((1, 3344, 1280, 1280, 5120), "mlp_flow_kernel"), ((1, 4080, 512, 224, 896), "mlp_tiles_kernel")])
def test_results_aligned_to_16_bytes_alone(cuda, shape, form):
    """The wave kernel writes 32 bytes at a time; results at other addresses come from the other forms, with the same bits."""
    batch, M, N, K, L = shape
    _, x, w1, w2, _ = _operands(cuda, *shape, torch.bfloat16, "IO", 52)
    want = ops.gemm_relu_gemm(x, w1, w2)
    out = torch.full((batch * M * N + 16,), float("nan"), dtype=torch.bfloat16, device=cuda)[8:8 + batch * M * N].view(batch, M, N)
    assert out.data_ptr() % 32 == 16
    ops.gemm_relu_gemm(x, w1, w2, out=out)
    assert torch.equal(out, want)
    assert form in _widths(lambda: ops.gemm_relu_gemm(x, w1, w2, out=out))


# cuts of the tile kernel that only calls have which else take the wave kernel: 256 columns for GEMM1, whole and in two parts, 192 of few tiles for GEMM2
@pytest.mark.parametrize("shape", [(1, 2064, 1024, 1024, 4096), (1, 2352, 768, 256, 3136), (1, 1376, 512, 8000, 1472), (1, 4096, 768, 768, 3072)])
@pytest.mark.parametrize("layout", ["IO", "OI"])
def test_tile_kernel_for_results_aligned_to_16_bytes_alone(cuda, shape, layout):
    batch, M, N, K, L = shape
    g, x, w1, w2, given = _operands(cuda, *shape, torch.bfloat16, layout, 54)
    out = torch.full((batch * M * N + 16,), float("nan"), dtype=torch.bfloat16, device=cuda)[8:8 + batch * M * N].view(batch, M, N)
    ops.gemm_relu_gemm(x, *given, out=out, weight_layout=layout)
    ref = torch.relu(x.float() @ w1.float()).to(torch.bfloat16).float() @ w2.float()
    _assert_close(out, ref, torch.bfloat16, shape, cuda)
    assert set(_widths(lambda: ops.gemm_relu_gemm(x, *given, out=out, weight_layout=layout))) == {"mlp_tiles_kernel"}
    b1, b2 = (torch.randn(batch, n, device=cuda, generator=g).to(torch.bfloat16) for n in (L, N))
    ops.ffn(x, given[0], b1, given[1], b2, out=out, act1="gelu", act2="identity", weight_layout=layout)
    h = _act(x.float() @ w1.float() + b1.float().view(batch, 1, L), "gelu").to(torch.bfloat16)
    _assert_close(out, h.float() @ w2.float() + b2.float().view(batch, 1, N), torch.bfloat16, ("ffn",) + shape, cuda)


def test_wave_kernel_streams_and_changed_weights(cuda):
    """The second launch reads its weights ahead of the first one's end: a weight written by the work just ahead in the
    stream is the one that is used, and calls on two streams have hidden layers of their own."""
    _, x, w1, w2, _ = _operands(cuda, 1, 4096, 768, 768, 3072, torch.bfloat16, "IO", 53)
    want = [ops.gemm_relu_gemm(x * s, w1 * s, w2 * s) for s in (1.0, 2.0, 0.5)]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    got = []
    for _ in range(6):
        for st in streams:
            with torch.cuda.stream(st):
                a, u, v = torch.empty_like(x), torch.empty_like(w1), torch.empty_like(w2)
                for i, s in enumerate((1.0, 2.0, 0.5)):
                    torch.mul(x, s, out=a), torch.mul(w1, s, out=u), torch.mul(w2, s, out=v)
                    got.append((ops.gemm_relu_gemm(a, u, v), want[i]))
    torch.cuda.synchronize()
    assert ops.device_status(cuda) == 0
    for g, w in got:
        assert torch.equal(g, w)
