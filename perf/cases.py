"""The work this package is used for, as cases that can be timed: fused attention chains, plain and ReLU GEMM
chains, feed-forward blocks and a whole transformer block, called the way a program calls them -- through
`ditto_b200.ops`, a module built from a chain definition, or a graph engine.

A case is a dict of plain values.  `kind` names the path:

  softmax   bmm -> softmax -> bmm, N and K up to 128
  chain     bmm -> bmm and bmm -> ReLU -> bmm, N and K up to 128
  mlp       GEMM -> ReLU -> GEMM with wide results, weights [in, out]
  ffn       feed-forward block with biases and two activations, weights [out, in]
  block     packed multi-head attention and the feed-forward block, run by a graph engine

`entry` is "ops" (a torch operator that allocates its result) or "module" (the built module that writes into the
caller's buffers, operands in the layout of the chain definition).
"""
import math

import torch

import ditto_b200 as ditto
from ditto_b200 import auto_compute as ac
from ditto_b200 import auto_schedule, auto_tensorize, chimera, hardware, ops, runtime
from ditto_b200.auto_compute.nn.model import TransformerBlock

_DTYPE = {"float16": torch.float16, "bfloat16": torch.bfloat16}


def listed():
    return [
        # one image through ViT-Base/16 (196 tokens padded to 208): the smallest call, all latency
        {"name": "vit-base-16-image", "kind": "softmax", "entry": "module", "batch": 12, "M": 208, "N": 64, "K": 64, "L": 208,
         "dtype": "float16", "layout": "KL", "scale": 1.0},
        # the plain chain on one Bert-Base sequence, through the built module
        {"name": "bert-base-chain", "kind": "chain", "entry": "module", "batch": 12, "M": 512, "N": 64, "K": 64, "L": 512,
         "dtype": "float16", "layout": "KL", "act": "identity"},
        # attention of one Bert-Base sequence: inference at batch 1
        {"name": "bert-base-sequence", "kind": "softmax", "entry": "ops", "batch": 12, "M": 512, "N": 64, "K": 64, "L": 512,
         "dtype": "float16", "layout": "LK", "scale": 0.125},
        # 16 images through ViT-Huge/16: head dimension 80, ragged rows
        {"name": "vit-huge-16-images", "kind": "softmax", "entry": "ops", "batch": 256, "M": 208, "N": 80, "K": 80, "L": 208,
         "dtype": "bfloat16", "layout": "LK", "scale": 80 ** -0.5},
        # 32 Bert-Large sequences: throughput at head dimension 64
        {"name": "bert-large-batch", "kind": "softmax", "entry": "ops", "batch": 512, "M": 512, "N": 64, "K": 64, "L": 512,
         "dtype": "float16", "layout": "LK", "scale": 0.125},
        # one long document, 16 heads of 64
        {"name": "long-document", "kind": "softmax", "entry": "ops", "batch": 16, "M": 8192, "N": 64, "K": 64, "L": 8192,
         "dtype": "float16", "layout": "LK", "scale": 0.125},
        # a batch of 64 long sequences, 16 heads of 128: the largest attention work
        {"name": "long-batch-d128", "kind": "softmax", "entry": "ops", "batch": 1024, "M": 2048, "N": 128, "K": 128, "L": 2048,
         "dtype": "bfloat16", "layout": "LK", "scale": 128 ** -0.5},
        # the feed-forward block of Bert-Base on one sequence: weights are most of what is read
        {"name": "ffn-bert-base-sequence", "kind": "ffn", "M": 512, "N": 768, "K": 768, "L": 3072, "dtype": "float16",
         "act1": "gelu", "act2": "identity"},
        # the feed-forward block of ViT-Huge on 16 images: a result wider than 1024 columns
        {"name": "ffn-vit-huge-images", "kind": "ffn", "M": 3328, "N": 1280, "K": 1280, "L": 5120, "dtype": "bfloat16",
         "act1": "gelu", "act2": "identity"},
        # the MLP chain on a few thousand rows: one of eight shards of the case below
        {"name": "mlp-2048-rows", "kind": "mlp", "M": 2048, "N": 1024, "K": 1024, "L": 4096, "dtype": "bfloat16", "act": "relu"},
        # the MLP chain on a training-size batch
        {"name": "mlp-16384-rows", "kind": "mlp", "M": 16384, "N": 1024, "K": 1024, "L": 4096, "dtype": "bfloat16", "act": "relu"},
        # a Bert-Base block on eight sequences, replayed by the engine as one CUDA graph
        {"name": "bert-base-block", "kind": "block", "batch": 8, "M": 512, "hidden": 768, "heads": 12, "ff": 3072,
         "dtype": "float16", "graph": True},
    ]


def _log16(rng, lo, hi):
    """A multiple of 16 between lo and hi, uniform over the logarithm."""
    return min(hi, max(lo, 16 * round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / 16)))


def _draw_small(rng, kind):
    """Attention and small chains: 1 to 1024 slices, 16 to 8192 rows and keys, widths 16 to 128 with 64 and 128
    the usual ones; mostly self-attention (as many keys as rows)."""
    while True:
        K = rng.choice([64, 64, 64, 128, 128, 80, 16 * rng.randint(1, 8)])
        N = K if rng.random() < 0.85 else 16 * rng.randint(1, 8)
        M = _log16(rng, 16, 8192)
        L = M if rng.random() < 0.7 else _log16(rng, 16, 8192)
        batch = round(math.exp(rng.uniform(0.0, math.log(1024))))
        if batch * M * L <= 1.6e9 and batch * (M + L) * (K + N) <= 5e8:
            break
    c = {"kind": kind, "entry": rng.choice(["ops", "module"]), "batch": batch, "M": M, "N": N, "K": K, "L": L,
         "dtype": rng.choice(["float16", "bfloat16"]), "layout": rng.choice(["KL", "LK"])}
    if c["entry"] == "module":
        c["dtype"], c["layout"] = "float16", "KL"
    if kind == "softmax":
        c["scale"] = 1.0 if c["entry"] == "module" else K ** -0.5
    else:
        c["act"] = "identity" if c["entry"] == "module" else rng.choice(["relu", "identity"])
    return c


def draw(rng):
    kind = rng.choice(["softmax"] * 5 + ["chain", "mlp", "mlp", "ffn", "ffn", "block"])
    if kind in ("softmax", "chain"):
        return _draw_small(rng, kind)
    if kind == "block":
        # hidden 256 to 1024 in heads of 64 or 128, one to 32 sequences of 64 to 1024 tokens
        d = rng.choice([64, 64, 128])
        hidden = 256 * rng.randint(1, 4)
        return {"kind": "block", "batch": round(math.exp(rng.uniform(0.0, math.log(32)))), "M": _log16(rng, 64, 1024),
                "hidden": hidden, "heads": hidden // d, "ff": 4 * hidden, "dtype": "float16", "graph": rng.random() < 0.5}
    # widths 256 to 2048, hidden layer mostly four times as wide, 16 to 16384 rows
    while True:
        N = 256 * rng.choice([1, 2, 3, 3, 4, 4, 4, 5, 6, 8])
        K = N if rng.random() < 0.75 else 16 * rng.randint(8, 128)
        L = 4 * N if rng.random() < 0.75 else 64 * rng.randint(4, 128)
        M = _log16(rng, 16, 16384)
        if 2.0 * M * L * (K + N) <= 3.5e11:
            break
    c = {"kind": kind, "M": M, "N": N, "K": K, "L": L, "dtype": rng.choice(["float16", "bfloat16"])}
    if kind == "mlp":
        c["act"] = rng.choice(["relu", "relu", "identity"])
    else:
        c["act1"], c["act2"] = rng.choice([("relu", "relu"), ("gelu", "identity"), ("relu", "identity")])
    return c


def _built_chain(case):
    """The call sequence of the front end, from the chain definition to the module."""
    F = ac.nn.functional
    define = F.BatchGemmSoftmaxGemm if case["kind"] == "softmax" else F.BatchGemmGemm
    ins, outs = define(case["batch"], case["M"], case["N"], case["K"], case["L"], case["dtype"], "float32")
    second = outs[0].op.input_tensors[0]
    first = second.op.input_tensors[0].op.input_tensors[0]
    b, m, n, mi, ni = second.op.axis
    rlo, rli = second.op.reduce_axis
    choice = auto_tensorize.fusion_choice(first.op, second.op, [b, m, n, rlo, mi, ni, rli], 3)
    info = {}
    for t, scope in ((first, "shared"), (second, "global")):
        packed = auto_tensorize.cuda_wmma(scope=scope)
        match = auto_tensorize.intrinsic_match(t, packed, ["InnerMost", "SameRange"])[0]
        info[t.op] = auto_tensorize.match_info(match, packed)
    layer = ac.layer([outs[0].op], inputs=ins)
    state = auto_tensorize.tensorize_hyper_fusion_state(layer, choice, info)
    sch = auto_tensorize.tensorize_cuda(layer, state, hardware.query_hw_param("gpu.cuda.B200"),
                                        auto_tensorize.cuda_tensorize_param())
    return ditto.build(sch, layer.schedule_tensors, "cuda")


def _built_block(case, normal):
    """Model -> graph -> fusion -> tasks -> schedules -> modules -> engine, with its weights in place."""
    hidden, ff, dtype = case["hidden"], case["ff"], case["dtype"]
    qkv = ac.layer_tensor([case["batch"], case["M"], 3 * hidden], name="qkv", dtype=dtype)
    model = TransformerBlock(hidden, case["heads"], ff, dtype=dtype, mma_in_dtype=dtype)
    graph = chimera.graph_fusion(ac.graph([qkv], [model(qkv)]))
    option = auto_schedule.ScheduleOption("cuda", device_name="gpu.cuda.B200", dtype=dtype, mma_in_dtype=dtype)
    bound = chimera.task_binding(auto_schedule.extract_tasks_from_graph(graph))
    schedules = auto_schedule.auto_schedule_bound_tasks(bound, option)
    built = {key: ditto.build(sch, args, "cuda") for key, (sch, args) in schedules.items()}
    make = runtime.create_cuda_graph_engine if case["graph"] else runtime.create_graph_engine
    engine = make(graph, built, "cuda")
    engine.get_function("init")()
    ffn = graph.all_layers[1]
    values = (normal(ff, hidden, std=hidden ** -0.5), normal(ff, std=0.5), normal(hidden, ff, std=ff ** -0.5),
              normal(hidden, std=0.5))
    for tensor, value in zip(ffn.weights, values):
        engine.get_function("set_weight")(ffn, tensor, value)
    engine.get_function("compile")()
    return engine


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    dtype = _DTYPE[case["dtype"]]

    def normal(*shape, std=1.0):
        t = torch.empty(shape, dtype=dtype, device="cuda")
        return t.normal_(0.0, std, generator=gen)

    def uniform(*shape):
        t = torch.empty(shape, dtype=dtype, device="cuda")
        return t.uniform_(-1.0, 1.0, generator=gen)

    kind = case["kind"]
    state = {"case": case}
    if kind == "block":
        # unscaled logits, as the layer defines them: half-size entries keep their spread at a few units
        state["qkv"] = normal(case["batch"], case["M"], 3 * case["hidden"], std=0.5)
        state["engine"] = _built_block(case, normal)
        return state
    M, N, K, L = case["M"], case["N"], case["K"], case["L"]
    if kind in ("softmax", "chain"):
        b = case["batch"]
        # the module takes the U(-1, 1) operands of the chain's own benchmark; the operators take attention's N(0, 1)
        make = uniform if case["entry"] == "module" or kind == "chain" else normal
        keys = (b, K, L) if case["layout"] == "KL" else (b, L, K)
        values = (b, N, L) if kind == "chain" and case["layout"] == "LK" else (b, L, N)
        state["tensors"] = (make(b, M, K), make(*keys), make(*values))
        if case["entry"] == "module":
            state["module"] = _built_chain(case)
            state["out"] = torch.empty(b, M, N, dtype=dtype, device="cuda")
    elif kind == "mlp":
        state["tensors"] = (normal(M, K), normal(K, L, std=K ** -0.5), normal(L, N, std=L ** -0.5))
    else:
        state["tensors"] = (normal(M, K), normal(L, K, std=K ** -0.5), normal(L, std=0.5), normal(N, L, std=L ** -0.5),
                            normal(N, std=0.5))
    return state


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "block":
        get = state["engine"].get_function
        get("set_inputs")(state["qkv"])
        get("run")()
        return get("get_outputs")()
    if case.get("entry") == "module":
        state["module"](*state["tensors"], state["out"])
        return state["out"]
    if kind == "softmax":
        return ops.bmm_softmax_bmm(*state["tensors"], scale=case["scale"], key_layout=case["layout"])
    if kind == "chain":
        # "KL" / "LK" name the layout of both weights here: [in, out] or [out, in]
        return ops.gemm_relu_gemm(*state["tensors"], activation=case["act"],
                                  weight_layout="IO" if case["layout"] == "KL" else "OI")
    if kind == "mlp":
        return ops.gemm_relu_gemm(*state["tensors"], activation=case["act"])
    return ops.ffn(*state["tensors"], act1=case["act1"], act2=case["act2"])


def work(case):
    """Every operand read once and every result written once, 16 bits each; two floating-point operations per
    multiply-add of the products (exponentials and activations are not counted)."""
    if case["kind"] == "block":
        rows, hidden, ff = case["batch"] * case["M"], case["hidden"], case["ff"]
        return {"bytes": 2.0 * (rows * 3 * hidden + 2 * hidden * ff + ff + hidden + rows * hidden),
                "flops": 4.0 * rows * case["M"] * hidden + 4.0 * rows * hidden * ff}
    b, M, N, K, L = case.get("batch", 1), case["M"], case["N"], case["K"], case["L"]
    biases = L + N if case["kind"] == "ffn" else 0
    return {"bytes": 2.0 * (b * (M * K + K * L + L * N + M * N) + biases), "flops": 2.0 * b * M * L * (K + N)}


def tolerance(case):
    """The intermediate and the result are rounded to the operand type (half an ulp: 2^-11 for fp16, 2^-8 / 2 for
    bf16), sums are 32-bit: two such implementations differ by about one rounding of each."""
    if case["dtype"] == "float16":
        return {"rel": 2e-3, "max": 2e-2}
    return {"rel": 1e-2, "max": 1e-1}
