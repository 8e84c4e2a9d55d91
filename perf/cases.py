"""The calls this library is used for on one GPU, at the sizes its configurations, tests and benchmark
name, as cases that can be timed: what a program has in hand beforehand (`prepare`), the call itself
(`run`), what the call cannot do without (`work`) and how far two correct results may lie apart
(`tolerance`).

Seven kinds of calls:

  allreduce   Communicator.all_reduce on device buffers: 8 KiB (latency) to 256 MiB (bandwidth), with the
              fused scale and the casts between bf16 and fp32 of the gradient path
  host        the same call on pinned host buffers, which is what the reference's own programs pass
  gemm        ops.gemm_bf16 in nn.Linear layout: few rows (decode), many rows (prefill), ragged shapes
  mlp         TensorParallelMLP.forward: all-gather -> GEMM with SwiGLU, GEMM -> reduce-scatter
  attn_out    TensorParallelAttnOut.forward: GEMM -> reduce-scatter
  local_sum   mncclLocalAllReduceNoAlloc: 2..4 buffers of one GPU, at most 64 KiB each
  ddp_step    DistributedDataParallel around the GPT-2 shaped decoder: forward, backward, bucket reduction
"""
import ctypes as C
import math

import torch

import mini_nccl_b200 as mn
from mini_nccl_b200.models import GPT2Config, GPT2Model
from mini_nccl_b200.ops import gemm_bf16
from mini_nccl_b200.parallel import DistributedDataParallel, TensorParallelAttnOut, TensorParallelMLP

TYPES = {"fp32": torch.float32, "bf16": torch.bfloat16, "fp16": torch.float16, "int32": torch.int32}
SIZES = {"fp32": 4, "bf16": 2, "fp16": 2, "int32": 4}
CODES = {"fp32": mn.FLOAT32, "bf16": mn.BFLOAT16, "fp16": mn.FLOAT16, "int32": mn.INT32}
OPS = {"sum": mn.SUM, "prod": mn.PROD, "max": mn.MAX, "min": mn.MIN, "avg": mn.AVG}

MAX_MESSAGE = 256 << 20           # bytes: the headline message
MAX_GEMM_FLOPS = 2.0 * 4096 * 14336 * 4096


def listed():
    return [
        # The smallest message of the AllReduce sweep: all latency (a norm, a loss, a small layer's gradient).
        {"name": "allreduce_8KiB_fp32", "kind": "allreduce", "count": 2048, "src": "fp32", "dst": "fp32", "scale": 1.0},
        # One 25 MB gradient bucket in bf16, averaged into its fp32 main-gradient buffer; a bucket's length is
        # whatever the parameters add up to, not a round number.
        {"name": "allreduce_25MB_bf16_to_fp32", "kind": "allreduce", "count": 13_106_408, "src": "bf16", "dst": "fp32",
         "scale": 0.125},
        # The headline message: 256 MiB of fp32, out of place.
        {"name": "allreduce_256MiB_fp32", "kind": "allreduce", "count": 64 << 20, "src": "fp32", "dst": "fp32", "scale": 1.0},
        # The reference's plumbing workload: 1,048,576 fp32 elements in host-mapped buffers.
        {"name": "host_4MiB_fp32", "kind": "host", "count": 1 << 20, "type": "fp32"},
        # The headline message end to end: input and result in pinned host memory.
        {"name": "host_256MiB_fp32", "kind": "host", "count": 64 << 20, "type": "fp32"},
        # Decode: a batch of 16 tokens through the FFN's first weight (hidden 4096, FFN 14336); weight traffic.
        {"name": "gemm_decode_16", "kind": "gemm", "m": 16, "n": 14336, "k": 4096, "out": "bf16"},
        # A ragged middle-sized product with an fp32 result: no dimension divides into tiles.
        {"name": "gemm_ragged_777", "kind": "gemm", "m": 777, "n": 1003, "k": 1544, "out": "fp32"},
        # Prefill: 4096 tokens through the same weight.
        {"name": "gemm_prefill_4096", "kind": "gemm", "m": 4096, "n": 14336, "k": 4096, "out": "bf16"},
        # One rank's share of the tensor-parallel MLP: 4096 tokens, hidden 4096, FFN 14336 over 8 ranks.
        {"name": "mlp_4096_tokens", "kind": "mlp", "tokens": 4096, "hidden": 4096, "ffn": 1792},
        # The attention output projection for a batch of 256 decode tokens.
        {"name": "attn_out_256_tokens", "kind": "attn_out", "tokens": 256, "hidden": 4096},
        # Four replicas' partial results of one GPU, 64 KiB each: the largest the entry point takes.
        {"name": "local_sum_4x64KiB", "kind": "local_sum", "buffers": 4, "count": 16384, "type": "fp32", "op": "sum"},
        # The data-parallel training step's gradient path: GPT-2-medium shape, micro-batch 8, 25 MB buckets.
        {"name": "ddp_gpt2_medium", "kind": "ddp_step", "layers": 24, "d_model": 1024, "vocab": 50257, "seq": 1024,
         "batch": 8, "main_grad": False},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _multiple(rng, lo, hi, step):
    return max(lo, _log_int(rng, lo, hi) // step * step)


def draw(rng):
    kind = rng.choice(["allreduce", "allreduce", "host", "gemm", "gemm", "mlp", "attn_out", "local_sum", "ddp_step"])
    if kind == "allreduce":
        src, dst = rng.choice([("fp32", "fp32"), ("bf16", "bf16"), ("bf16", "fp32"), ("fp32", "bf16"), ("fp16", "fp16"),
                               ("int32", "int32")])
        count = _log_int(rng, 2048, MAX_MESSAGE // max(SIZES[src], SIZES[dst]))
        scale = 1.0 if src == "int32" else rng.choice([1.0, 0.5, 0.125])
        return {"kind": kind, "count": count, "src": src, "dst": dst, "scale": scale}
    if kind == "host":
        t = rng.choice(["fp32", "bf16"])
        return {"kind": kind, "count": _log_int(rng, 2048, MAX_MESSAGE // SIZES[t]), "type": t}
    if kind == "gemm":
        while True:
            m, n = _log_int(rng, 1, 8192), _log_int(rng, 64, 14336)
            if rng.random() < 0.5:
                n = max(64, n // 64 * 64)          # a layer's width more often than not divides into tiles
            k = _multiple(rng, 64, 14336, 8)
            if 2.0 * m * n * k <= MAX_GEMM_FLOPS:
                return {"kind": kind, "m": m, "n": n, "k": k, "out": rng.choice(["bf16", "bf16", "fp32"])}
    if kind == "mlp":
        return {"kind": kind, "tokens": _multiple(rng, 128, 4096, 128), "hidden": _multiple(rng, 512, 4096, 64),
                "ffn": _multiple(rng, 256, 3584, 16)}
    if kind == "attn_out":
        return {"kind": kind, "tokens": _multiple(rng, 128, 4096, 128), "hidden": _multiple(rng, 512, 4096, 64)}
    if kind == "local_sum":
        t = rng.choice(["fp32", "bf16", "fp16", "int32"])
        return {"kind": kind, "buffers": rng.choice([2, 3, 4]), "count": _log_int(rng, 64, (64 << 10) // SIZES[t]), "type": t,
                "op": rng.choice(["sum", "avg", "max"])}
    return {"kind": kind, "layers": _log_int(rng, 2, 24), "d_model": 64 * _log_int(rng, 2, 16),
            "vocab": _log_int(rng, 512, 50257), "seq": _multiple(rng, 64, 1024, 8), "batch": rng.randint(1, 8),
            "main_grad": rng.random() < 0.5}


def _values(gen, count, name):
    """normal(0, 1) as the sweep's inputs; integers of a counter's size."""
    if name == "int32":
        return torch.randint(-100000, 100000, (count,), generator=gen, device="cuda", dtype=torch.int32)
    return torch.randn(count, generator=gen, device="cuda").to(TYPES[name])


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    kind, state = case["kind"], {"case": case}
    if kind == "gemm":
        state["a"] = torch.randn(case["m"], case["k"], generator=gen, device="cuda").to(torch.bfloat16)
        state["b"] = (torch.randn(case["n"], case["k"], generator=gen, device="cuda") * 0.02).to(torch.bfloat16)
        state["out_dtype"] = TYPES[case["out"]]
        return state
    if kind == "local_sum":
        n = case["buffers"]
        state["send"] = [_values(gen, case["count"], case["type"]) for _ in range(n)]
        state["recv"] = [torch.zeros_like(t) for t in state["send"]]
        state["send_ptrs"] = (C.c_void_p * n)(*[t.data_ptr() for t in state["send"]])
        state["recv_ptrs"] = (C.c_void_p * n)(*[t.data_ptr() for t in state["recv"]])
        state["args"] = (n, case["count"], CODES[case["type"]], OPS[case["op"]])
        fn = mn.lib().mncclLocalAllReduceNoAlloc
        fn.restype = C.c_int
        fn.argtypes = [C.POINTER(C.c_void_p), C.POINTER(C.c_void_p), C.c_int, C.c_size_t, C.c_int, C.c_int, C.c_void_p]
        state["fn"] = fn
        return state
    comm = state["comm"] = mn.Communicator(1, 0)
    if kind == "allreduce":
        state["x"] = _values(gen, case["count"], case["src"])
        state["y"] = torch.empty(case["count"], dtype=TYPES[case["dst"]], device="cuda")
    elif kind == "host":
        # pinned buffers live as long as the program and the data arrive in them
        state["x"] = torch.empty(case["count"], dtype=TYPES[case["type"]], pin_memory=True)
        state["x"].copy_(_values(gen, case["count"], case["type"]))
        state["y"] = torch.empty(case["count"], dtype=TYPES[case["type"]], pin_memory=True)
    elif kind == "mlp":
        mlp = state["block"] = TensorParallelMLP(comm, case["tokens"], case["hidden"], case["ffn"], seed=seed)
        # the previous layer writes its activations straight into the gather buffer
        mlp.input_shard.copy_(torch.randn(case["tokens"], case["hidden"], generator=gen, device="cuda") * 0.5)
    elif kind == "attn_out":
        state["block"] = TensorParallelAttnOut(comm, case["tokens"], case["hidden"], seed=seed)
        state["x"] = (torch.randn(case["tokens"], case["hidden"], generator=gen, device="cuda") * 0.5).to(torch.bfloat16)
    else:
        torch.manual_seed(seed)
        cfg = GPT2Config(n_layer=case["layers"], d_model=case["d_model"], n_head=case["d_model"] // 64,
                         vocab_size=case["vocab"], seq_len=case["seq"])
        with torch.device("cuda"):
            model = GPT2Model(cfg).to(torch.bfloat16)
        state["ddp"] = DistributedDataParallel(model, comm, bucket_mb=25.0,
                                               main_grad_dtype=torch.float32 if case["main_grad"] else None)
        state["ids"] = torch.randint(0, case["vocab"], (case["batch"], case["seq"]), generator=gen, device="cuda")
    return state


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "allreduce":
        return state["comm"].all_reduce(state["x"], "sum", out=state["y"], scale=case["scale"])
    if kind == "host":
        return state["comm"].all_reduce(state["x"], "sum", out=state["y"])
    if kind == "gemm":
        return gemm_bf16(state["a"], state["b"], out_dtype=state["out_dtype"])
    if kind == "mlp":
        return state["block"].forward()
    if kind == "attn_out":
        return state["block"].forward(state["x"])
    if kind == "local_sum":
        rc = state["fn"](state["send_ptrs"], state["recv_ptrs"], *state["args"], torch.cuda.current_stream().cuda_stream)
        if rc != 0:
            raise RuntimeError("mncclLocalAllReduceNoAlloc: %d" % rc)
        return state["recv"]
    ddp = state["ddp"]
    ddp.zero_grad()
    loss = ddp(state["ids"], state["ids"])
    loss.backward()
    return [loss.detach()] + [b.flat if b.main is None else b.main for b in ddp.buckets]


def work(case):
    kind = case["kind"]
    if kind == "allreduce":
        return {"bytes": case["count"] * (SIZES[case["src"]] + SIZES[case["dst"]]), "flops": 0}
    if kind == "host":
        return {"bytes": 2 * case["count"] * SIZES[case["type"]], "flops": 0}
    if kind == "gemm":
        m, n, k = case["m"], case["n"], case["k"]
        return {"bytes": 2 * (m * k + n * k) + SIZES[case["out"]] * m * n, "flops": 2.0 * m * n * k}
    if kind == "mlp":
        t, h, f = case["tokens"], case["hidden"], case["ffn"]
        return {"bytes": 2 * (2 * t * h + 3 * h * f), "flops": 6.0 * t * h * f}
    if kind == "attn_out":
        t, h = case["tokens"], case["hidden"]
        return {"bytes": 2 * (2 * t * h + h * h), "flops": 2.0 * t * h * h}
    if kind == "local_sum":
        n, size = case["buffers"], SIZES[case["type"]]
        return {"bytes": 2 * n * case["count"] * size, "flops": (n - 1) * case["count"]}
    # The parameters are read forward and backward and their gradients written; a causal attention's two
    # products cover half of the square.
    d, layers, tokens = case["d_model"], case["layers"], case["batch"] * case["seq"]
    matrices = layers * 12 * d * d + case["vocab"] * d
    attention = layers * 2 * 2.0 * tokens * case["seq"] * d / 2
    params = matrices + case["seq"] * d
    return {"bytes": 2 * params * (3 + (2 if case["main_grad"] else 0)), "flops": 6.0 * matrices * tokens + 3 * attention}


def tolerance(case):
    kind = case["kind"]
    if kind in ("allreduce", "host", "local_sum"):
        # one rank: a product with the scale, rounded once; several buffers: added in buffer order in fp32
        return "exact"
    if kind == "gemm":
        # fp32 sums in another order; for bf16 a last rounding that may fall the other way
        return {"rel": 1e-5} if case["out"] == "fp32" else {"rel": 4e-3}
    if kind in ("mlp", "attn_out"):
        return {"rel": 1e-2}
    # bf16 activations and gradients through many layers, and an attention backward whose sums have no fixed order
    return {"rel": 2e-2, "max": 0.9}
