"""Large calls of the MLP chain where there is no memory for their whole hidden layer: they take the ring that serves the flow kernel, as a
caller's workspace of that size does, and go without scratch memory only where there is none for the ring either."""
import pytest
import torch

from ditto_b200 import _lib, ops


class _Sizes:
    """A library that asks for `full` bytes, or for `ring` where there is no memory for them."""

    def __init__(self, full, ring):
        self.full, self.ring = full, ring

    def ditto_b200_workspace_bytes(self, op, *shape):
        return self.ring if op & _lib.OP_LESS_SCRATCH else self.full


@pytest.mark.parametrize("full,ring,room,got", [(1000, 300, 2000, 1000), (1000, 300, 999, 300), (1000, 300, 299, 0), (1000, 0, 999, 0), (0, 0, 2000, 0)])
def test_sizes_that_are_tried(monkeypatch, full, ring, room, got):
    empty = torch.empty

    def short(n, **more):
        if n > room:
            raise torch.OutOfMemoryError("no memory")
        return empty(n, **more)

    monkeypatch.setattr(torch, "empty", short)
    buf, ptr, size = ops._scratch(_Sizes(full, ring), _lib.OP_GEMM_RELU_GEMM, 1, 16, 256, 128, 64, torch.float16, torch.device("cpu"))
    assert size == got and (buf is None) == (got == 0) and (got == 0) == (ptr is None)
    assert buf is None or (buf.numel() == got and buf.data_ptr() == ptr)


SHAPE = (1, 65552, 256, 128, 1024)         # a hidden layer of 128 MB


def _operands(cuda):
    _, M, N, K, L = SHAPE
    g = torch.Generator(device=cuda).manual_seed(52)
    x, w1 = torch.randn(M, K, device=cuda, generator=g).half(), (torch.randn(K, L, device=cuda, generator=g) * K ** -0.5).half()
    w2, b1 = (torch.randn(L, N, device=cuda, generator=g) * L ** -0.5).half(), torch.randn(L, device=cuda, generator=g).half()
    return x, w1, b1, w2


@pytest.mark.gpu
def test_less_scratch_is_the_ring(cuda):
    need = _lib.load().ditto_b200_workspace_bytes
    op = _lib.OP_GEMM_RELU_GEMM
    ring = need(op | _lib.EPILOGUE_FLOW_MMA, *SHAPE, 0)
    assert 0 < need(op | _lib.OP_LESS_SCRATCH, *SHAPE, 0) == ring < need(op, *SHAPE, 0)
    # calls of the tile and the cluster kernels have no size in between, nor calls whose ring holds the whole hidden layer, nor calls by name
    for shape in ((1, 512, 768, 768, 3072), (64, 128, 1024, 512, 4096), (24, 384, 768, 768, 3072), (1, 65552, 256, 64, 1024), (1, 64, 64, 64, 64)):
        assert need(op | _lib.OP_LESS_SCRATCH, *shape, 0) == 0
    assert need(op | _lib.OP_LESS_SCRATCH | _lib.EPILOGUE_WIDE_MMA, *SHAPE, 0) == 0


@pytest.mark.gpu
def test_large_calls_take_the_ring_where_memory_is_short(cuda):
    """On the native and on the checked path, with room for the ring and not for the hidden layer: the ring is what is taken (the
    allocator counts it), and the result is that of a caller's workspace of that size."""
    x, w1, b1, w2 = _operands(cuda)
    need = _lib.load().ditto_b200_workspace_bytes
    full, ring = need(_lib.OP_GEMM_RELU_GEMM, *SHAPE, 0), need(_lib.OP_GEMM_RELU_GEMM | _lib.EPILOGUE_FLOW_MMA, *SHAPE, 0)
    assert ring + (24 << 20) < full
    want = ops.gemm_relu_gemm(x, w1, w2, workspace=torch.empty(ring, dtype=torch.uint8, device=cuda))
    assert torch.equal(want, ops.gemm_relu_gemm(x, w1, w2, variant="flow"))
    out, block = torch.empty_like(want), torch.empty_like(want)
    fast, total = ops._fast, torch.cuda.get_device_properties(cuda).total_memory
    assert fast is not None
    taken = []
    try:
        for path in (fast, None):
            ops._fast = path
            for call in (lambda: ops.gemm_relu_gemm(x, w1, w2, out=out),
                         lambda: ops.ffn(x, w1, b1, w2, None, out=block, act1="relu", act2="identity", weight_layout="IO")):
                torch.cuda.synchronize()
                torch.cuda.empty_cache()
                torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + ring + (24 << 20)) / total)
                before = torch.cuda.memory_stats()
                call()
                call()
                after = torch.cuda.memory_stats()
                taken.append(after["allocated_bytes.all.allocated"] - before["allocated_bytes.all.allocated"])
                # no request failed: the allocator would have given its cached blocks back, waiting for the device, in every call
                assert (after["num_ooms"], after["num_alloc_retries"]) == (before["num_ooms"], before["num_alloc_retries"])
            assert torch.equal(out, want)
            h = torch.relu(x[:4096].float() @ w1.float() + b1.float()).half().float()
            torch.testing.assert_close(block[:4096].float(), h @ w2.float(), rtol=2 ** -9, atol=2e-3)
            out.zero_(), block.zero_()
    finally:
        ops._fast = fast
        torch.cuda.set_per_process_memory_fraction(1.0)
    assert ops.device_status(cuda) == 0
    assert all(2 * ring <= n < 2 * ring + (8 << 20) for n in taken), (ring, full, taken)
