"""The attention kernel with 64-key blocks (head dimensions up to 64), against float64 products of the same 16-bit operands:
one to many blocks, partial last blocks, row tails, widths below 64, both layouts and types, packed heads, the chains
without a softmax, growing maxima and scores of -inf; and large calls, which take it by themselves."""
import pytest
import torch

from ditto_b200 import _lib, ops
from tests.test_gpu_attention_split import _close, _reference

pytestmark = pytest.mark.gpu

NARROW = _lib.FLAG_NARROW


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("b,M,N,K,L,layout", [
    (3, 128, 64, 64, 64, "LK"),        # one block
    (2, 144, 64, 64, 16, "KL"),        # a block of 16 keys, a row tail
    (3, 16, 64, 64, 128, "LK"),        # two blocks: no stage is refilled
    (2, 208, 64, 64, 208, "KL"),       # four, the last of 16 keys
    (1, 272, 48, 16, 1168, "LK"),      # widths below 64
    (2, 128, 16, 64, 320, "KL"),
    (40, 2048, 64, 64, 80, "LK"),      # more CTAs than the device holds at once
])
def test_shapes(dtype, b, M, N, K, L, layout):
    g = torch.Generator(device="cuda").manual_seed(b * M + L)
    q = torch.randn(b, M, K, generator=g, device="cuda").to(dtype)
    k = torch.randn(b, L, K, generator=g, device="cuda").to(dtype)
    v = torch.randn(b, L, N, generator=g, device="cuda").to(dtype)
    keys = k if layout == "LK" else k.transpose(1, 2).contiguous()
    out = ops.bmm_softmax_bmm(q, keys, v, scale=2 * K ** -0.5, key_layout=layout, flags=NARROW)
    assert ops.device_status() == 0
    _close(out, _reference(q, k, v, 2 * K ** -0.5), dtype)
    assert torch.equal(out, ops.bmm_softmax_bmm(q, keys, v, scale=2 * K ** -0.5, key_layout=layout, flags=NARROW))


def test_growing_maxima_and_infinite_scores():
    g = torch.Generator(device="cuda").manual_seed(6)
    b, M, d, L = 1, 128, 64, 512
    q = (torch.rand(b, M, d, generator=g, device="cuda") + 0.5).bfloat16()
    v = torch.randn(b, L, d, generator=g, device="cuda").bfloat16()
    k = torch.randn(b, L, d, generator=g, device="cuda").bfloat16()
    k = (k.float() * (1 + torch.arange(L, device="cuda")[None, :, None] / 40)).bfloat16()      # the maximum grows past the rescale threshold
    _close(ops.bmm_softmax_bmm(q, k, v, scale=0.5, key_layout="LK", flags=NARROW), _reference(q, k, v, 0.5), torch.bfloat16)
    for lo, hi in ((0, 64), (128, 512)):               # q is positive: scores of -inf for whole blocks, the first or the last
        ki = k.clone()
        ki[:, lo:hi] = float("-inf")
        rest = [i for i in range(L) if not lo <= i < hi]
        _close(ops.bmm_softmax_bmm(q, ki, v, scale=0.25, key_layout="LK", flags=NARROW),
               _reference(q, k[:, rest], v[:, rest], 0.25), torch.bfloat16)
    assert ops.device_status() == 0


@pytest.mark.parametrize("heads,d,M", [(4, 64, 1040), (3, 48, 80)])
def test_packed_heads(heads, d, M):
    g = torch.Generator(device="cuda").manual_seed(M)
    qkv = torch.randn(2, M, 3 * heads * d, generator=g, device="cuda").half()
    out = ops.multi_head_attention(qkv, heads, scale=d ** -0.5, flags=NARROW)
    assert ops.device_status() == 0
    for i in range(2):
        q, k, v = (t.reshape(M, heads, d).transpose(0, 1) for t in qkv[i].chunk(3, dim=-1))
        _close(out[i], _reference(q, k, v, d ** -0.5).transpose(0, 1).reshape(M, heads * d), torch.float16)


@pytest.mark.parametrize("act", ["identity", "relu"])
@pytest.mark.parametrize("layout", ["IO", "OI"])
@pytest.mark.parametrize("b,M,N,K,L", [(600, 144, 64, 64, 208), (300, 512, 32, 48, 256), (320, 16, 64, 64, 64)])
def test_many_items_of_a_chain(act, layout, b, M, N, K, L):
    g = torch.Generator(device="cuda").manual_seed(M + L)
    x = torch.randn(b, M, K, generator=g, device="cuda").half()
    w1 = (torch.randn(b, K, L, generator=g, device="cuda") * K ** -0.5).half()
    w2 = (torch.randn(b, L, N, generator=g, device="cuda") * L ** -0.5).half()
    h = x.float() @ w1.float()
    want = ((h.relu() if act == "relu" else h).half().float() @ w2.float()).double()
    ws = (w1, w2) if layout == "IO" else (w1.transpose(1, 2).contiguous(), w2.transpose(1, 2).contiguous())
    out = ops.gemm_relu_gemm(x, *ws, activation=act, weight_layout=layout)
    assert ops.device_status() == 0
    _close(out, want, torch.float16)


@pytest.mark.parametrize("b,M,L", [(20, 2048, 2048), (320, 128, 512), (150, 512, 208), (60, 2048, 2064)])
def test_many_items(b, M, L):
    g = torch.Generator(device="cuda").manual_seed(b)
    q = torch.randn(b, M, 64, generator=g, device="cuda").half()
    k = torch.randn(b, L, 64, generator=g, device="cuda").half()
    v = torch.randn(b, L, 64, generator=g, device="cuda").half()
    out = ops.bmm_softmax_bmm(q, k, v, scale=0.125, key_layout="LK")
    assert ops.device_status() == 0
    for i in range(0, b, 7):
        _close(out[i:i + 1], _reference(q[i:i + 1], k[i:i + 1], v[i:i + 1], 0.125), torch.float16)


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("L", [144, 208, 512])
def test_no_less_precise_than_longer_blocks(L, dtype):
    """The norm of the error against float64 beside that of the kernel with 128-key blocks, from flat to peaked rows.  The
    error is the rounding of some 10^6 results and 10^8 weights, so that two kernels of the same precision differ by
    less than 1 %."""
    g = torch.Generator(device="cuda").manual_seed(L)
    b, M, d = 64, 256, 64
    q = torch.randn(b, M, d, generator=g, device="cuda").to(dtype)
    k = torch.randn(b, L, d, generator=g, device="cuda").to(dtype)
    v = torch.randn(b, L, d, generator=g, device="cuda").to(dtype)
    for scale in (0.0625, 0.125, 0.2, 0.35, 0.6, 1.0):
        want = _reference(q, k, v, scale)
        narrow, whole = ((ops.bmm_softmax_bmm(q, k, v, scale=scale, key_layout="LK", flags=f).double() - want).norm().item()
                         for f in (NARROW, _lib.FLAG_SPLIT_UNIT))
        assert narrow <= 1.01 * whole, (scale, narrow / want.norm().item(), whole / want.norm().item())


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
def test_weights_far_apart_and_scores_that_are_not_numbers(dtype):
    """Weights come from two pipes, by a key's place in the block: both give 2^x down to where it is nothing, 0 for -inf and NaN for
    NaN.  A row's tolerance is _close's (rounding of the weights and of the result); exponents differ by up to 2^-13 (kFusedReference)."""
    g = torch.Generator(device="cuda").manual_seed(9)
    b, M, d, L = 1, 128, 64, 128
    q = torch.ones(b, M, d, device="cuda", dtype=dtype)
    v = torch.randn(b, L, d, generator=g, device="cuda").to(dtype)
    # scores d * x with x from 0 to -3.5: weights 1 to 2^-320, in an order that gives every place in a block all sizes
    for turn in range(4):
        x = torch.linspace(0, -3.5, L, device="cuda").roll(17 * turn)[torch.randperm(L, generator=g, device="cuda")]
        k = x[None, :, None].expand(b, L, d).to(dtype).contiguous()
        _close(ops.bmm_softmax_bmm(q, k, v, key_layout="LK", flags=NARROW), _reference(q, k, v, 1.0), dtype)
    k = torch.randn(b, L, d, generator=g, device="cuda").to(dtype)
    for key in list(range(16)) + [63, 64, 127]:
        for bad, place in ((float("nan"), k), (float("inf"), k)):
            broken = place.clone()
            broken[0, key] = bad
            assert torch.isnan(ops.bmm_softmax_bmm(q, broken, v, scale=0.125, key_layout="LK", flags=NARROW)).all(), (key, bad)
        gone = k.clone()
        gone[0, key] = float("-inf")
        rest = [i for i in range(L) if i != key]
        _close(ops.bmm_softmax_bmm(q, gone, v, scale=0.125, key_layout="LK", flags=NARROW), _reference(q, k[:, rest], v[:, rest], 0.125), dtype)
    assert ops.device_status() == 0


@pytest.mark.parametrize("on_fma", [0, 1])
def test_exponentials_by_themselves(on_fma):
    """Both pipes against float64: 2^-22 of the value, which is ex2.approx's bound, and the polynomial no further off than ex2.approx was
    measured to be (1.45e-7); 0 from -127 on (below -126 values are no normal numbers and a pipe may give 0) and for -inf, NaN for NaN."""
    lib = _lib.load()

    def ex2(x):
        y = torch.full_like(x, float("nan"))
        assert lib.ditto_b200_selftest_ex2(x.data_ptr(), y.data_ptr(), x.numel(), on_fma, torch.cuda.current_stream().cuda_stream) == 0
        return y
    for lo, hi in ((-126, 127), (-30, 9), (-1, 1), (-2 ** -10, 2 ** -10)):
        x = torch.linspace(lo, hi, 1 << 22, device="cuda", dtype=torch.float64).float()
        assert ((ex2(x).double() / torch.exp2(x.double()) - 1).abs().max()) <= (1.45e-7 if on_fma else 2 ** -22), (lo, hi)
    x = torch.arange(-126, 128, device="cuda").float()
    assert torch.equal(ex2(x).double(), torch.exp2(x.double()))
    x = torch.linspace(-127, -126, 4096, device="cuda")
    assert (ex2(x).double() - torch.exp2(x.double())).abs().max() <= 2 ** -126
    low = torch.tensor([-127.0, -127.5, -128.0, -150.0, -1e4, -3e38, -1e30, float("-inf")], device="cuda")
    assert torch.equal(ex2(low), torch.zeros_like(low))
    assert ex2(torch.full((2,), float("nan"), device="cuda")).isnan().all()
