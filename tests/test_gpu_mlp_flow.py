"""The two-GEMM flow kernel (the form of the MLP chain that is given scratch memory) at the sizes where it can go
wrong, against float32 products.  Bounds: those of the random-shape sweeps, one rounding of the hidden layer and one
of the result at the operand type's precision plus a floor scaled by the largest result."""
import pytest
import torch

from ditto_b200 import _lib, ops
from tests.test_gpu_random_shapes import _act, _assert_close

pytestmark = pytest.mark.gpu

# one 16-row tile and a split hidden dimension; a second CTA with 80 rows and a K tail; a second row block of 16 rows;
# one hidden tile of 64 columns; a single last chunk in a round (1088 = 4 x 256 + 64); a result of five tiles; three
# batch entries with partial blocks; more row blocks than the ring of hidden tiles holds; an odd number of k-steps
SHAPES = ((1, 16, 1024, 128, 4096), (1, 208, 256, 80, 512), (1, 272, 512, 64, 2048), (1, 128, 256, 64, 64),
          (1, 256, 512, 192, 1088), (1, 336, 1280, 96, 768), (3, 400, 512, 64, 1024), (1, 256 * 41 + 16, 256, 64, 1024),
          (2, 2064, 768, 320, 3072))


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("layout", ["IO", "OI"])
@pytest.mark.parametrize("form", ["relu", "identity", "relu+relu", "gelu+none", "relu+none", "gelu+relu, one bias"])
def test_flow_kernel(cuda, dtype, layout, form):
    g = torch.Generator(device=cuda).manual_seed(31)
    lib = _lib.load()
    for (batch, M, N, K, L) in SHAPES:
        assert lib.ditto_b200_workspace_bytes(_lib.OP_GEMM_RELU_GEMM, batch, M, N, K, L, 0) > 0
        if form not in ("relu", "identity") and batch > 1:
            continue
        x = torch.randn(batch, M, K, device=cuda, generator=g).to(dtype)
        w1 = (torch.randn(batch, K, L, device=cuda, generator=g) * K ** -0.5).to(dtype)
        w2 = (torch.randn(batch, L, N, device=cuda, generator=g) * L ** -0.5).to(dtype)
        a1, a2 = (w1.transpose(1, 2).contiguous(), w2.transpose(1, 2).contiguous()) if layout == "OI" else (w1, w2)
        out = torch.full((batch, M, N), float("nan"), dtype=dtype, device=cuda)
        if form in ("relu", "identity"):
            ops.gemm_relu_gemm(x, a1, a2, out=out, activation=form, weight_layout=layout)
            ref = _act(x.float() @ w1.float(), form).to(dtype).float() @ w2.float()
        else:
            acts = {"relu+relu": ("relu", "relu"), "gelu+none": ("gelu", "identity"), "relu+none": ("relu", "identity")}.get(form, ("gelu", "relu"))
            b1 = (torch.randn(1, L, device=cuda, generator=g) * 0.5).to(dtype)
            b2 = None if "one bias" in form else (torch.randn(1, N, device=cuda, generator=g) * 0.5).to(dtype)
            ops.ffn(x, a1, b1, a2, b2, out=out, act1=acts[0], act2=acts[1], weight_layout=layout)
            y = _act(x.float() @ w1.float() + b1.float()[:, None, :], acts[0]).to(dtype).float() @ w2.float()
            ref = _act(y if b2 is None else y + b2.float()[:, None, :], acts[1])
        _assert_close(out, ref, dtype, (form, batch, M, N, K, L, str(dtype), layout), cuda)


def test_flow_kernel_runs_are_identical_and_streams_do_not_mix(cuda):
    """Scratch memory arrives dirty and is per call: repeated calls give the same bits, on one stream and on two whose
    launches overlap (split hidden ranges and shared row blocks of the ring included)."""
    g = torch.Generator(device=cuda).manual_seed(32)
    data = []
    for M in (48, 2048):
        x = torch.randn(M, 512, device=cuda, generator=g).bfloat16()
        w1 = (torch.randn(512, 4096, device=cuda, generator=g) * 512 ** -0.5).bfloat16()
        w2 = (torch.randn(4096, 512, device=cuda, generator=g) * 4096 ** -0.5).bfloat16()
        data.append((x, w1, w2, ops.gemm_relu_gemm(x, w1, w2)))
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    outs = []
    for _ in range(10):
        for s, (x, w1, w2, want) in zip(streams, data):
            with torch.cuda.stream(s):
                outs.append((ops.gemm_relu_gemm(x, w1, w2), want))
    torch.cuda.synchronize()
    assert ops.device_status(cuda) == 0
    for got, want in outs:
        assert torch.equal(got, want)


def test_flow_kernel_needs_its_scratch_memory(cuda):
    """A workspace that is too small is not an error: the call takes the kernel that keeps the hidden layer in a cluster."""
    g = torch.Generator(device=cuda).manual_seed(33)
    x = torch.randn(256, 128, device=cuda, generator=g).bfloat16()
    w1 = (torch.randn(128, 2048, device=cuda, generator=g) * 128 ** -0.5).bfloat16()
    w2 = (torch.randn(2048, 256, device=cuda, generator=g) * 2048 ** -0.5).bfloat16()
    small = ops.gemm_relu_gemm(x, w1, w2, workspace=torch.empty(1024, dtype=torch.uint8, device=cuda))
    assert torch.equal(small, ops.gemm_relu_gemm(x, w1, w2, workspace=None))
    need = _lib.load().ditto_b200_workspace_bytes(_lib.OP_GEMM_RELU_GEMM, 1, 256, 256, 128, 2048, _lib.DTYPE_BF16)
    dirty = torch.full((need,), 0xA5, dtype=torch.uint8, device=cuda)
    assert torch.equal(ops.gemm_relu_gemm(x, w1, w2, workspace=dirty), ops.gemm_relu_gemm(x, w1, w2))


def test_search_for_a_plan_is_short_and_kept(cuda):
    """The host's share of a large call: the search for a shape that is new, batches of thousands of entries included, and
    the look-up of one that a few hundred other shapes were called after.  (48 us and under 1 us; the limits leave room for a busy host.)"""
    import time
    lib = _lib.load()
    shapes = [(b, M, N, N, 4 * N) for b, M in ((1, 16384), (1, 8208), (24, 384), (512, 256), (2048, 160), (1, 131072)) for N in (512, 1024)]
    shapes += [(1, 16384 + 16 * i, 1024, 1024, 4096) for i in range(60)]
    call = lambda b, M, N, K, L: lib.ditto_b200_workspace_bytes(_lib.OP_GEMM_RELU_GEMM | _lib.EPILOGUE_FLOW_MMA, b, M, N, K, L, 1)     # noqa: E731
    call(1, 4096, 512, 512, 2048)                          # (the kernel's attributes are set here)
    times = []
    for _ in range(2):
        times.append([])
        for s in shapes:
            t = time.perf_counter()
            assert call(*s) > 0
            times[-1].append(time.perf_counter() - t)
    assert sorted(times[0])[-3] < 1e-3, sorted(times[0])[-5:]
    assert sorted(times[1])[len(shapes) // 2] < 20e-6, times[1]
