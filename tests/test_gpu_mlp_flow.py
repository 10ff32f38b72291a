"""The two-GEMM flow kernel at the sizes where it can go wrong, against float32 products.  Large calls with scratch memory take
it by rule; small ones are asked for by name, and the feed-forward block, which names no kernel, is made large by its hidden
layer alone.  Bounds: those of the random-shape sweeps, one rounding of the hidden layer and one of the result at the operand
type's precision plus a floor scaled by the largest result."""
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


# hidden layers beyond what the tile kernel takes, at widths that cost little: a second CTA with 16 rows and one k-step; batch
# entries with partial row blocks and a K tail; a last chunk of 64 columns and more row blocks than the ring holds
LARGE = ((1, 24592, 256, 16, 1024), (3, 8208, 256, 80, 1024), (1, 24656, 512, 48, 1088))


def _takes_flow(batch, M, N, K, L):
    """Whether the rules on sizes give a call with scratch memory to the flow kernel: its scratch memory is the flow kernel's."""
    need = _lib.load().ditto_b200_workspace_bytes
    return need(_lib.OP_GEMM_RELU_GEMM, batch, M, N, K, L, 0) == need(_lib.OP_GEMM_RELU_GEMM | _lib.EPILOGUE_FLOW_MMA, batch, M, N, K, L, 0) \
        != batch * M * L * 2


def _operands(cuda, batch, M, N, K, L, dtype, layout, seed):
    g = torch.Generator(device=cuda).manual_seed(seed)
    x = torch.randn(batch, M, K, device=cuda, generator=g).to(dtype)
    w1 = (torch.randn(batch, K, L, device=cuda, generator=g) * K ** -0.5).to(dtype)
    w2 = (torch.randn(batch, L, N, device=cuda, generator=g) * L ** -0.5).to(dtype)
    given = (w1.transpose(1, 2).contiguous(), w2.transpose(1, 2).contiguous()) if layout == "OI" else (w1, w2)
    return g, x, w1, w2, given


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("layout", ["IO", "OI"])
@pytest.mark.parametrize("act", ["relu", "identity"])
def test_flow_kernel(cuda, dtype, layout, act):
    for shape in SHAPES:
        _, x, w1, w2, given = _operands(cuda, *shape, dtype, layout, 31)
        out = torch.full((shape[0], shape[1], shape[2]), float("nan"), dtype=dtype, device=cuda)
        ops.gemm_relu_gemm(x, *given, out=out, activation=act, weight_layout=layout, variant="flow")
        ref = _act(x.float() @ w1.float(), act).to(dtype).float() @ w2.float()
        _assert_close(out, ref, dtype, (act, shape, str(dtype), layout), cuda)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("layout", ["IO", "OI"])
@pytest.mark.parametrize("form", ["relu+relu", "gelu+identity", "relu+identity", "gelu+relu", "relu+relu, first bias", "gelu+identity, second bias",
                                  "relu+identity, misaligned", "identity+gelu, none"])
def test_flow_kernel_with_biases(cuda, dtype, layout, form):
    """The epilogues known at compile time and those picked at run time: a bias missing, biases at addresses that allow no 16-byte loads."""
    acts, _, which = form.partition(", ")
    act1, act2 = acts.split("+")
    for shape in LARGE:
        batch, M, N, K, L = shape
        assert _takes_flow(*shape)
        g, x, w1, w2, given = _operands(cuda, *shape, dtype, layout, 32)
        off = 2 if which == "misaligned" else 0
        bias = (torch.randn(batch * (L + N) + 16, device=cuda, generator=g) * 0.5).to(dtype)
        b1 = None if which in ("second bias", "none") else bias[off:off + batch * L].view(batch, L)
        b2 = None if which in ("first bias", "none") else bias[off + batch * L:off + batch * (L + N)].view(batch, N)
        out = torch.full((batch, M, N), float("nan"), dtype=dtype, device=cuda)
        ops.ffn(x, given[0], b1, given[1], b2, out=out, act1=act1, act2=act2, weight_layout=layout)
        h = x.float() @ w1.float() + (0 if b1 is None else b1.float()[:, None])
        y = _act(h, act1).to(dtype).float() @ w2.float() + (0 if b2 is None else b2.float()[:, None])
        _assert_close(out, _act(y, act2), dtype, (form, shape, str(dtype), layout), cuda)


def test_flow_kernel_runs_are_identical_and_streams_do_not_mix(cuda):
    """Scratch memory arrives dirty and is per call: repeated calls give the same bits, on one stream and on two whose
    launches overlap (a hidden dimension split in three, one split in two, and more row blocks than the ring holds)."""
    g = torch.Generator(device=cuda).manual_seed(32)
    data = []
    for M, L in ((48, 4096), (2048, 4096), (16400, 2048)):
        x = torch.randn(M, 512, device=cuda, generator=g).bfloat16()
        w1 = (torch.randn(512, L, device=cuda, generator=g) * 512 ** -0.5).bfloat16()
        w2 = (torch.randn(L, 512, device=cuda, generator=g) * L ** -0.5).bfloat16()
        data.append((x, w1, w2, ops.gemm_relu_gemm(x, w1, w2, variant="flow")))
    ring_bytes = _lib.load().ditto_b200_workspace_bytes(_lib.OP_GEMM_RELU_GEMM | _lib.EPILOGUE_FLOW_MMA, 1, 16400, 512, 512, 2048, 1)
    assert ring_bytes < 16400 * 2048 * 2
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    outs = []
    for i in range(12):
        for s, (x, w1, w2, want) in zip(streams, (data[i % 3], data[(i + 1) % 3])):
            with torch.cuda.stream(s):
                outs.append((ops.gemm_relu_gemm(x, w1, w2, variant="flow"), want))
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
    need = _lib.load().ditto_b200_workspace_bytes
    for variant, bit in (("auto", 0), ("flow", _lib.EPILOGUE_FLOW_MMA)):
        n = need(_lib.OP_GEMM_RELU_GEMM | bit, 1, 256, 256, 128, 2048, _lib.DTYPE_BF16)
        dirty = torch.full((n,), 0xA5, dtype=torch.uint8, device=cuda)
        assert torch.equal(ops.gemm_relu_gemm(x, w1, w2, workspace=dirty, variant=variant), ops.gemm_relu_gemm(x, w1, w2, variant=variant))
    with pytest.raises(RuntimeError):                      # by name there is no other kernel to take
        ops.gemm_relu_gemm(x, w1, w2, variant="flow", workspace=None)


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
