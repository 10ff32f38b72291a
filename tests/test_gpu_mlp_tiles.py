"""The tile kernel, which small calls of the MLP chain with scratch memory take, at the sizes where it can go wrong, against
float32 products (bounds as in the random-shape sweeps): all its tile widths, reduction splits and epilogues; and the rules
on sizes that choose between it, the flow kernel and the cluster kernels."""
import pytest
import torch

from ditto_b200 import _lib, ops
from tests.test_gpu_random_shapes import _act, _assert_close

pytestmark = pytest.mark.gpu


def _operands(cuda, batch, M, N, K, L, dtype, seed):
    g = torch.Generator(device=cuda).manual_seed(seed)
    x = torch.randn(batch, M, K, device=cuda, generator=g).to(dtype)
    w1 = (torch.randn(batch, K, L, device=cuda, generator=g) * K ** -0.5).to(dtype)
    w2 = (torch.randn(batch, L, N, device=cuda, generator=g) * L ** -0.5).to(dtype)
    return g, x, w1, w2


@pytest.mark.parametrize("layout", ["IO", "OI"])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_large_calls(cuda, dtype, layout):
    # large enough for the flow kernel
    for batch, M, N, K, L in ((1, 3344, 1280, 1280, 5120), (1, 16400, 512, 512, 2048)):
        _, x, w1, w2 = _operands(cuda, batch, M, N, K, L, dtype, 41)
        a1, a2 = (w1, w2) if layout == "IO" else (w1.transpose(1, 2).contiguous(), w2.transpose(1, 2).contiguous())
        for act in ("relu", "identity"):
            out = ops.gemm_relu_gemm(x, a1, a2, activation=act, weight_layout=layout)
            assert torch.equal(out, ops.gemm_relu_gemm(x, a1, a2, activation=act, weight_layout=layout, variant="flow"))
            ref = _act(x.float() @ w1.float(), act).to(dtype).float() @ w2.float()
            _assert_close(out, ref, dtype, (act, batch, M, N, K, L, str(dtype), layout), cuda)


# one k-step in either GEMM; a last tile wider than what is left of the result (256, 192 and 128 columns); two CTAs per SM over
# several waves; a K tail; batches with partial row blocks; 256 columns in two parts, with an odd number of chunks to divide, and
# of entries with partial row blocks; clusters of two, four and eight for either GEMM (test_cabi.py sees that all cuts are here)
SHAPES = ((1, 16, 256, 16, 64), (1, 16, 1024, 1024, 4096), (1, 144, 256, 4096, 128), (1, 512, 768, 768, 3072),
          (1, 2064, 1024, 1024, 4096), (1, 8208, 256, 272, 1088), (1, 4096, 768, 768, 3072), (5, 80, 512, 144, 576),
          (1, 1040, 2048, 512, 2112), (1, 2352, 768, 256, 3136), (2, 608, 1280, 128, 5120), (1, 512, 1024, 1024, 4096),
          (1, 16, 256, 2624, 6272), (2, 16, 2048, 16, 1536), (1, 16, 512, 1216, 3456), (1, 544, 1280, 48, 1856),
          (1, 32, 256, 5488, 64), (1, 16, 256, 2112, 3328), (1, 1376, 512, 8000, 1472), (3, 1168, 1024, 16, 320))


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("layout", ["IO", "OI"])
@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_tile_kernel(cuda, shape, layout, dtype):
    batch, M, N, K, L = shape
    g, x, w1, w2 = _operands(cuda, batch, M, N, K, L, dtype, 43)
    a1, a2 = (w1, w2) if layout == "IO" else (w1.transpose(1, 2).contiguous(), w2.transpose(1, 2).contiguous())
    assert _lib.load().ditto_b200_workspace_bytes(_lib.OP_GEMM_RELU_GEMM, batch, M, N, K, L, 0) == batch * M * L * 2
    out = ops.gemm_relu_gemm(x, a1, a2, weight_layout=layout)
    ref = torch.relu(x.float() @ w1.float()).to(dtype).float() @ w2.float()
    _assert_close(out, ref, dtype, ("chain",) + shape, cuda)
    assert torch.equal(out, ops.gemm_relu_gemm(x, a1, a2, weight_layout=layout))
    # biases at addresses that allow 16-byte loads and at such that do not, and one bias missing
    bias = (torch.randn(batch * (L + N) + 2, device=cuda, generator=g) * 0.5).to(dtype)
    for b1, b2 in ((bias[:batch * L], bias[batch * L:batch * (L + N)]), (bias[2:2 + batch * L], None),
                   (None, bias[2:2 + batch * N])):
        out = ops.ffn(x, a1, b1, a2, b2, act1="gelu", act2="relu", weight_layout=layout)
        h = x.float() @ w1.float() + (0 if b1 is None else b1.float().view(batch, 1, L))
        y = _act(h, "gelu").to(dtype).float() @ w2.float() + (0 if b2 is None else b2.float().view(batch, 1, N))
        _assert_close(out, _act(y, "relu"), dtype, ("ffn",) + shape, cuda)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_cuts_differ_by_the_order_of_sums_alone(cuda, dtype):
    """Operands whose sums are whole numbers below 2^24: any order gives the same bits, those of the call without scratch memory and
    of float64 products, however a reduction is divided."""
    for batch, M, N, K, L in SHAPES + ((1, 2048, 1024, 1024, 4096),):
        g = torch.Generator(device=cuda).manual_seed(46)
        x, w1, w2 = (torch.randint(-a, a + 1, size, device=cuda, generator=g).to(dtype)
                     for a, size in ((2, (batch, M, K)), (1, (batch, K, L)), (2, (batch, L, N))))
        h = torch.relu(x.double() @ w1.double()).to(dtype)
        sums = h.double() @ w2.double()
        assert 2 * h.double().sum(dim=-1).max() < 2 ** 24 and 2 * x.abs().double().sum(dim=-1).max() < 2 ** 24
        want = sums.float().to(dtype)
        assert torch.equal(ops.gemm_relu_gemm(x, w1, w2), want), (batch, M, N, K, L)
        assert torch.equal(ops.gemm_relu_gemm(x, w1, w2, workspace=None), want), (batch, M, N, K, L)


def test_tile_kernel_streams_and_changed_weights(cuda):
    """The second launch reads its weights ahead of the first one's end: a weight written by the work just ahead in the
    stream is the one that is used, and calls on two streams have hidden layers of their own."""
    _, x, w1, w2 = _operands(cuda, 1, 512, 768, 768, 3072, torch.bfloat16, 44)
    want = [ops.gemm_relu_gemm(x * s, w1 * s, w2 * s) for s in (1.0, 2.0, 0.5)]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    got = []
    for _ in range(10):
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


@pytest.mark.parametrize("shape,form", [
    ((64, 128, 1024, 512, 4096), _lib.EPILOGUE_WIDE_MMA),     # entries of one 128-row block, whole rounds of clusters
    ((33, 336, 1024, 256, 4096), _lib.EPILOGUE_WIDE_MMA),     # three of them
    ((40, 128, 1024, 1024, 4096), "tiles"),                   # a second round of seven clusters only
    ((60, 112, 1280, 256, 5120), "tiles"),                    # a width the cluster kernel computes in two groups
    ((520, 128, 256, 64, 1024), "tiles"),                     # a hidden layer larger than L2
    ((400, 128, 512, 64, 2048), _lib.EPILOGUE_WIDE_MMA),      # ... and wide enough for the cluster kernel
    ((24, 384, 768, 768, 3072), _lib.EPILOGUE_FLOW_MMA),      # a quarter of the flow kernel's rows are zero
    ((16, 512, 1024, 1024, 4096), _lib.EPILOGUE_FLOW_MMA),
])
def test_form_of_batched_calls(cuda, shape, form):
    """Rules on sizes for weights of every entry's own (seen by the scratch memory asked for), and the form's result."""
    batch, M, N, K, L = shape
    need = _lib.load().ditto_b200_workspace_bytes
    want = batch * M * L * 2 if form == "tiles" else need(_lib.OP_GEMM_RELU_GEMM | form, *shape, 1)
    assert need(_lib.OP_GEMM_RELU_GEMM, *shape, 1) == want
    _, x, w1, w2 = _operands(cuda, batch, M, N, K, L, torch.bfloat16, 45)
    out = ops.gemm_relu_gemm(x, w1, w2)
    for i in (0, batch // 2, batch - 1):
        ref = torch.relu(x[i].float() @ w1[i].float()).bfloat16().float() @ w2[i].float()
        _assert_close(out[i], ref, torch.bfloat16, shape, cuda)
