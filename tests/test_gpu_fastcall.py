"""The native call path against the checked Python path: the same calls give the same bits and shapes, and what the checked
path refuses is refused with its errors, whichever path saw the call first."""
import ctypes
import threading

import pytest
import torch

from ditto_b200 import _lib, ops

pytestmark = pytest.mark.gpu


def _both(fn):
    """Results (or error types) of the native and of the checked path."""
    got = []
    fast = ops._fast
    for path in (fast, None):
        ops._fast = path
        try:
            got.append(fn())
        except Exception as e:                          # noqa: BLE001 - the error is the result
            got.append((type(e), str(e)))
        finally:
            ops._fast = fast
    return got


def _t(*shape, dtype=torch.float16, device="cuda"):
    return torch.randn(*shape, device=device).to(dtype)


def _calls():
    q, k, v = _t(2, 144, 64), _t(2, 272, 64), _t(2, 272, 48)
    x, w1, w2 = _t(48, 128), _t(128, 320), _t(320, 256)
    qkv = _t(2, 64, 3 * 128)
    yield "softmax", lambda: ops.bmm_softmax_bmm(q, k, v, scale=0.125, key_layout="LK")
    yield "integer scale and flags", lambda: ops.bmm_softmax_bmm(q, k, v, scale=1, key_layout="LK", flags=2)
    yield "given result", lambda: ops.bmm_softmax_bmm(q, k, v, out=torch.empty(2, 144, 48, device="cuda", dtype=q.dtype),
                                                      scale=0.125, key_layout="LK")
    yield "heads", lambda: ops.multi_head_attention(qkv, 2, scale=0.5)
    yield "chain", lambda: ops.gemm_relu_gemm(x, w1, w2)
    yield "batched chain", lambda: ops.gemm_relu_gemm(x[None], w1[None], w2[None], activation="identity")
    yield "flat result of a batch of one", lambda: ops.gemm_relu_gemm(x[None], w1[None], w2[None],
                                                                      out=torch.empty(48, 256, device="cuda", dtype=x.dtype))
    yield "no scratch", lambda: ops.gemm_relu_gemm(x, w1, w2, workspace=None)
    yield "ffn", lambda: ops.ffn(x, w1, _t(320) * 0 + 1, w2, None, act1="gelu", act2="identity", weight_layout="IO")
    yield "requires grad", lambda: ops.gemm_relu_gemm(x.clone().requires_grad_(), w1, w2)
    # refused
    yield "wrong key layout", lambda: ops.bmm_softmax_bmm(q, k, v, key_layout="KL")
    yield "unknown layout", lambda: ops.bmm_softmax_bmm(q, k, v, key_layout="XX")
    yield "float32", lambda: ops.bmm_softmax_bmm(q.float(), k.float(), v.float(), key_layout="LK")
    yield "mixed types", lambda: ops.bmm_softmax_bmm(q, k.bfloat16(), v, key_layout="LK")
    yield "host tensor", lambda: ops.bmm_softmax_bmm(q.cpu(), k, v, key_layout="LK")
    yield "not a tensor", lambda: ops.bmm_softmax_bmm([1], k, v, key_layout="LK")
    yield "strided", lambda: ops.bmm_softmax_bmm(q.transpose(0, 1), k, v, key_layout="LK")
    yield "wrong result shape", lambda: ops.bmm_softmax_bmm(q, k, v, out=torch.empty_like(q), key_layout="LK")
    yield "text scale", lambda: ops.bmm_softmax_bmm(q, k, v, scale="x", key_layout="LK")
    yield "negative scale", lambda: ops.bmm_softmax_bmm(q, k, v, scale=-1.0, key_layout="LK")
    yield "rows not of 16", lambda: ops.bmm_softmax_bmm(q[:, :100].contiguous(), k, v, key_layout="LK")
    yield "misaligned", lambda: ops.gemm_relu_gemm(_t(48 * 128 + 1)[1:].view(48, 128), w1, w2)
    yield "empty", lambda: ops.gemm_relu_gemm(x[:0], w1, w2)
    yield "heads that do not divide", lambda: ops.multi_head_attention(qkv, 5)
    yield "no heads", lambda: ops.multi_head_attention(qkv, 0)
    yield "unknown activation", lambda: ops.gemm_relu_gemm(x, w1, w2, activation="gelu")
    yield "short bias", lambda: ops.ffn(x, w1, _t(319), w2, None, weight_layout="IO")


class _Recorder:
    """The native module, noting what its functions answered."""

    def __init__(self, module):
        self.module, self.answers = module, []

    def __getattr__(self, name):
        def call(*args):
            self.answers.append(getattr(self.module, name)(*args))
            return self.answers[-1]
        return call


def test_native_path_answers_like_the_checked_path(cuda):
    """... and answers itself where the call is valid, and not at all where it is refused."""
    ops.bmm_softmax_bmm(_t(1, 16, 16), _t(1, 16, 16), _t(1, 16, 16), key_layout="LK")     # sets the native path up
    assert ops._fast is not None
    torch.manual_seed(3)
    fast = ops._fast
    for name, call in _calls():
        ops._fast = recorder = _Recorder(fast)
        try:
            native, checked = _both(call)
        finally:
            ops._fast = fast
        assert len(recorder.answers) == 1, name
        if isinstance(checked, tuple):
            assert native == checked and recorder.answers == [None], name
        else:
            assert recorder.answers[0] is native, name
            assert native.shape == checked.shape and native.dtype == checked.dtype and torch.equal(native, checked), name
    assert ops.device_status(cuda) == 0


def _modules():
    """Built modules of every kind with valid arguments, results last."""
    from ditto_b200.auto_tensorize import ChainSchedule
    from ditto_b200.runtime.module import ChainModule

    def module(kind, batch, M, N, K, L, **more):
        return ChainModule(ChainSchedule(layer=None, kind=kind, batch=batch, M=M, N=N, K=K, L=L, dtype="float16", device=None,
                                         param=None, **{"scale": 1.0, **more}))

    b, M, N, K, L = 2, 48, 64, 32, 80
    chain = (_t(b, M, K), _t(b, K, L), _t(b, L, N), _t(b, M, N))
    for kind in ("softmax", "relu", "identity"):
        yield module(kind, b, M, N, K, L), chain
    yield module("mha", 2, 48, 64, 32, 48, heads=2, scale=0.5), (_t(2, 48, 192), _t(2, 48, 64))
    M, N, K, L = 48, 256, 128, 320
    x, w1, b1, w2, b2, y = _t(M, K), _t(L, K), _t(L), _t(N, L), _t(N), _t(M, N)
    for bias1, bias2 in ((0, 0), (1, 0), (0, 1), (1, 1)):
        args = (x, w1, *((b1,) if bias1 else ()), w2, *((b2,) if bias2 else ()), y)
        yield module("ffn", 1, M, N, K, L, bias1=bool(bias1), bias2=bool(bias2), act1="gelu", act2="relu"), args


def test_modules_answer_in_native_code(cuda):
    """Every kind of module: the second call is the native one, with the bits of the first; wrong arguments are refused by it and
    reported by the checked path."""
    torch.manual_seed(6)
    for module, args in _modules():
        what = (module.schedule.kind, len(args))
        module(*args)                                       # the checked path
        want = args[-1].clone()
        args[-1].zero_()
        assert ops._fast.call(module._plan, *args) is True, what
        assert torch.equal(args[-1], want), what
        for i in range(len(args)):
            for bad in (args[i][..., :-16].contiguous(), args[i].bfloat16(), args[i].cpu()):
                wrong = args[:i] + (bad,) + args[i + 1:]
                assert ops._fast.call(module._plan, *wrong) is None, (what, i)
                with pytest.raises((TypeError, ValueError)):
                    module(*wrong)
        assert ops._fast.call(module._plan, *args[:-1]) is None, what
        with pytest.raises(TypeError):
            module(*args[:-1])
    assert ops.device_status(cuda) == 0


def test_entry_points_run_without_the_interpreter_lock(cuda):
    """With each C entry point replaced by PyGILState_Check -- 0, a successful call, where the calling thread does not hold the lock."""
    q, x, w1, w2, qkv = _t(1, 16, 16), _t(16, 128), _t(128, 64), _t(64, 256), _t(1, 16, 48)
    ops.bmm_softmax_bmm(q, q, q, key_layout="LK")
    fast, lib = ops._fast, _lib.load()
    address = lambda fn: ctypes.cast(fn, ctypes.c_void_p).value                       # noqa: E731
    own = [address(getattr(lib, "ditto_b200_" + n)) for n in ("bmm_softmax_bmm", "multi_head_attention", "gemm_relu_gemm", "ffn_ws", "workspace_bytes")]
    check = address(ctypes.pythonapi.PyGILState_Check)
    ab, a2 = torch.empty(16, 256, device=cuda, dtype=x.dtype), torch.empty(1, 16, 16, device=cuda, dtype=x.dtype)
    fp16 = ops._DTYPE_CODE[x.dtype]
    plans = [(fast.plan(0, 1, 16, 16, 16, 16, fp16, 1, 1.0, 0, 0, 0, 0), (q, q, q, a2)),
             (fast.plan(1, 1, 16, 16, 16, 16, fp16, 1, 1.0, 1, 0, 0, 0), (q, q, q, a2)),
             (fast.plan(2, 1, 16, 16, 16, 16, fp16, 1, 1.0, 0, 0, 0, 0), (qkv, a2)),
             (fast.plan(3, 1, 16, 256, 128, 64, fp16, 1, 1.0, 1, 0, 0, 0), (x, w1.T.contiguous(), w2.T.contiguous(), ab))]
    fast.bind(check, check, check, check, own[4])
    try:
        got = [fast.softmax(q, q, q, None, 1.0, "LK", 0), fast.mha(qkv, 1, None, 1.0, 0),
               fast.gemm(x, w1, w2, None, "relu", "IO", True), fast.ffn(x, w1, None, w2, None, None, "relu", "relu", "IO")]
        called = [fast.call(plan, *tensors) for plan, tensors in plans]
    finally:
        fast.bind(*own)
    assert all(isinstance(t, torch.Tensor) for t in got)
    assert called == [True] * 4


def test_two_threads(cuda):
    """Calls from two threads, each on a stream of its own, give the bits of calls in turn."""
    torch.manual_seed(4)
    work = []
    for M in (144, 272):
        q, x, w1, w2 = _t(6, M, 64), _t(M, 256), _t(256, 1024) / 16, _t(1024, 256) / 32
        calls = (lambda q=q: ops.bmm_softmax_bmm(q, q, q, scale=0.125, key_layout="LK"),
                 lambda x=x, u=w1, v=w2: ops.gemm_relu_gemm(x, u, v), lambda x=x, u=w1, v=w2: ops.ffn(x, u, None, v, None, weight_layout="IO"))
        work.append([(c, c()) for c in calls])
    torch.cuda.synchronize()
    wrong = []

    def run(items):
        with torch.cuda.stream(torch.cuda.Stream()):
            for _ in range(50):
                got = [c() for c, _ in items]
            torch.cuda.current_stream().synchronize()
            wrong.extend(i for i, (g, (_, want)) in enumerate(zip(got, items)) if not torch.equal(g, want))

    threads = [threading.Thread(target=run, args=(items,)) for items in work]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong and ops.device_status(cuda) == 0
