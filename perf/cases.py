"""Performance cases: the work a program built on mccl_b200 has one GPU do, through the package's public entry points.

A case is a dict with a "kind" and its sizes.  `listed()` gives the fixed set, `draw(rng)` one more case of the same
ranges, `prepare` what the program has in hand before the call, `run` one pass, `work` the bytes and operations a pass
cannot do without, `tolerance` how far two correct implementations of the same precision may differ.

    step        one data-parallel training step of the GPT-2 style decoder: forward, backward, gradient norm, clipped AdamW
    logits      forward pass of the same model without gradients (scoring a batch)
    llama       forward and backward of the tensor-parallel decoder on a communicator of one rank
    mlp         forward and backward of the tensor-parallel SiLU MLP whose forward runs in the fused GEMM kernels
    moe         forward and backward of the expert-parallel layer with the fused dispatch and combine
    gemm        the tcgen05 matrix product, plain or with SiLU in its epilogue
    loss        softmax cross-entropy over bf16 logits, forward and backward
    norm        LayerNorm, forward and backward
    optim       gradient norm and clipped AdamW over one flat bucket
    collective  all-reduce, reduce-scatter and all-gather on a communicator of one rank
"""
from __future__ import annotations

import math

import torch

import mccl_b200 as mccl
from mccl_b200.models.gpt2 import GPT2, GPT2Config
from mccl_b200.models.llama import Llama, LlamaConfig
from mccl_b200.ops.gemm import gemm
from mccl_b200.ops.loss import fused_cross_entropy
from mccl_b200.ops.norm import FusedLayerNorm
from mccl_b200.ops.optim import fused_adamw_, scratch_floats, sum_squares_
from mccl_b200.parallel.ddp import DistributedDataParallel
from mccl_b200.parallel.layers import ExpertParallelMoE
from mccl_b200.parallel.tp import FusedTensorParallelMLP

DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32, "int32": torch.int32}



def listed():
    return [
        # The smallest model the package configures, one step issued call by call: what a step costs before any size
        # matters (a first run, a unit test, a small model): launches and host time.
        {"name": "step_tiny_eager", "kind": "step", "layers": 2, "d_model": 128, "heads": 4, "ffn": 512, "vocab": 1000, "seq": 64,
         "batch": 4, "graph": False},
        # The workload of bench.py: 24 layers, width 1024, 8 sequences of 1024 tokens, the step replayed from a CUDA graph.
        {"name": "step_medium_graph", "kind": "step", "layers": 24, "d_model": 1024, "heads": 16, "ffn": 4096, "vocab": 50257,
         "seq": 1024, "batch": 8, "graph": True},
        # Scoring a few sequences of uneven length with the same model family: forward only, rows no tile divides.
        {"name": "logits_ragged", "kind": "logits", "layers": 12, "d_model": 768, "heads": 12, "ffn": 3072, "vocab": 50257,
         "seq": 777, "batch": 3},
        # Pre-training the tensor-parallel decoder: its default vocabulary and sequence, half its default width, two blocks
        # (every block is the same work).
        {"name": "llama_step", "kind": "llama", "layers": 2, "d_model": 2048, "heads": 16, "ffn": 5504, "vocab": 32000, "seq": 2048,
         "batch": 2},
        # One MLP of a tensor-parallel model in training, at the sizes of the eight-GPU test.
        {"name": "mlp_8192", "kind": "mlp", "tokens": 8192, "hidden": 2048, "ffn": 8192},
        # One expert layer in training: eight experts, a quarter of spare capacity, so some slots stay empty and
        # crowded experts drop tokens.
        {"name": "moe_8_experts", "kind": "moe", "tokens": 8192, "hidden": 1024, "ffn": 2048, "experts": 8, "spare": 0.25},
        # A narrow batch through one projection, rows that only the one-SM form takes: few tiles, latency counts.
        {"name": "gemm_small", "kind": "gemm", "m": 384, "n": 1024, "k": 1024, "silu": False},
        # The up projection of the fused FFN at the size the kernels' benchmark uses.
        {"name": "gemm_large_silu", "kind": "gemm", "m": 8192, "n": 3584, "k": 8192, "silu": True},
        # The loss of the benchmark's training step: 8192 tokens, vocabulary padded to a multiple of 64 columns.
        {"name": "loss_8192", "kind": "loss", "rows": 8192, "vocab": 50257, "padded": True},
        # The norms of a medium model on an uneven batch.
        {"name": "norm_ragged", "kind": "norm", "rows": 5003, "d": 1024},
        # One gradient bucket of the default size (25 MB of bf16) with a few elements over, as the flat buckets have.
        {"name": "optim_bucket", "kind": "optim", "elems": 25 * (1 << 20) // 2 + 5, "clip": True},
        # Small messages on a communicator of one rank (a program written for n GPUs run on one): the call's latency.
        {"name": "collective_small", "kind": "collective", "elems": 16384, "dtype": "bf16", "op": "avg"},
    ]


# ---- drawing --------------------------------------------------------------------------------------------------------
def _log_int(rng, lo, hi, step=1):
    """A multiple of `step` in [lo, hi], uniform in its logarithm."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return max(lo, min(hi, int(round(v / step)) * step))


def _decoder(rng):
    d = rng.choice([128, 256, 384, 512, 640, 768, 1024])
    return {"layers": _log_int(rng, 1, 24), "d_model": d, "heads": d // rng.choice([32, 64]), "ffn": 4 * d,
            "vocab": _log_int(rng, 1000, 50257), "seq": _log_int(rng, 48, 1024), "batch": rng.randint(1, 8)}


def draw(rng):
    kind = rng.choice(["step", "step", "logits", "llama", "mlp", "moe", "gemm", "gemm", "loss", "norm", "optim", "collective"])
    if kind == "step":
        return {"kind": kind, **_decoder(rng), "graph": rng.random() < 0.5}
    if kind == "logits":
        return {"kind": kind, **_decoder(rng)}
    if kind == "llama":
        d = rng.choice([256, 512, 1024, 1536, 2048])
        return {"kind": kind, "layers": rng.randint(1, 2), "d_model": d, "heads": d // rng.choice([64, 128]),
                "ffn": _log_int(rng, 2 * d, 5504, 64) if 2 * d < 5504 else 5504, "vocab": _log_int(rng, 256, 32000),
                "seq": _log_int(rng, 32, 2048), "batch": rng.randint(1, 2)}
    if kind == "mlp":
        return {"kind": kind, "tokens": _log_int(rng, 128, 8192, 128), "hidden": _log_int(rng, 256, 2048, 64),
                "ffn": _log_int(rng, 512, 8192, 64)}
    if kind == "moe":
        return {"kind": kind, "tokens": _log_int(rng, 64, 8192), "hidden": _log_int(rng, 128, 1024, 8),
                "ffn": _log_int(rng, 256, 2048, 8), "experts": rng.choice([2, 4, 8, 16, 32]), "spare": rng.choice([0.0, 0.25, 1.0])}
    if kind == "gemm":
        return {"kind": kind, "m": _log_int(rng, 128, 8192, 128), "n": _log_int(rng, 64, 3584, 64), "k": _log_int(rng, 64, 8192, 64),
                "silu": rng.random() < 0.5}
    if kind == "loss":
        vocab = _log_int(rng, 256, 131072)
        return {"kind": kind, "rows": _log_int(rng, 1, min(16384, 8192 * 50257 // vocab)), "vocab": vocab,
                "padded": rng.random() < 0.6}
    if kind == "norm":
        return {"kind": kind, "rows": _log_int(rng, 1, 32768), "d": rng.choice([128, 256, 384, 512, 768, 1024, 2048])}
    if kind == "optim":
        return {"kind": kind, "elems": _log_int(rng, 1024, 64 << 20), "clip": rng.random() < 0.7}
    return {"kind": kind, "elems": _log_int(rng, 16, 64 << 20), "dtype": rng.choice(list(DTYPES)), "op": rng.choice(["sum", "avg", "max"])}


# ---- what the program has in hand -----------------------------------------------------------------------------------
_comm = None


def _one_rank():
    """The program's communicator (one rank), created once per process as a program does."""
    global _comm
    if _comm is None:
        torch.cuda.set_device(0)
        _comm = mccl.Communicator(1, mccl.get_unique_id(), 0, transport="cuda")
    return _comm


def _tokens(case, gen):
    t = torch.randint(0, case["vocab"], (case["batch"], case["seq"] + 1), device="cuda", generator=gen)
    return t[:, :-1].contiguous(), t[:, 1:].contiguous()


def _gpt2(case):
    cfg = GPT2Config(n_layer=case["layers"], d_model=case["d_model"], n_head=case["heads"], d_ff=case["ffn"],
                     vocab_size=case["vocab"], seq_len=case["seq"])
    with torch.device("cuda"):
        return GPT2(cfg).to(torch.bfloat16)


def prepare(case, seed):
    torch.manual_seed(seed)                                    # the models' initial weights
    gen = torch.Generator(device="cuda").manual_seed(seed)     # everything else

    def normal(*shape, std=1.0, mean=0.0):
        return (torch.randn(*shape, device="cuda", generator=gen) * std + mean).to(torch.bfloat16)

    kind, s = case["kind"], {"kind": case["kind"]}
    if kind == "step":
        s["idx"], s["targets"] = _tokens(case, gen)
        s["ddp"] = DistributedDataParallel(_gpt2(case), None)
        s["replay"] = s["ddp"].graphed_step((s["idx"], s["targets"]), lr=3e-4, max_grad_norm=1.0) if case["graph"] else None
    elif kind == "logits":
        s["idx"], _ = _tokens(case, gen)
        s["model"] = _gpt2(case)
    elif kind == "llama":
        s["idx"], s["targets"] = _tokens(case, gen)
        cfg = LlamaConfig(n_layer=case["layers"], d_model=case["d_model"], n_head=case["heads"], d_ff=case["ffn"],
                          vocab_size=case["vocab"], seq_len=case["seq"])
        with torch.device("cuda"):
            s["model"] = Llama(cfg, _one_rank()).to(torch.bfloat16)
        torch.nn.init.normal_(s["model"].embed.weight, std=0.02)
    elif kind == "mlp":
        s["layer"] = FusedTensorParallelMLP(_one_rank(), case["tokens"], case["hidden"], case["ffn"])
        s["x"] = normal(case["tokens"], case["hidden"]).requires_grad_(True)
        s["dy"] = normal(case["tokens"], case["hidden"], std=1e-2)
    elif kind == "moe":
        capacity = math.ceil(case["tokens"] / case["experts"] * (1 + case["spare"]))
        s["layer"] = ExpertParallelMoE(_one_rank(), case["hidden"], case["ffn"], case["experts"], capacity, device="cuda",
                                       dtype=torch.bfloat16, fused=True)
        s["x"] = normal(case["tokens"], case["hidden"]).requires_grad_(True)
        s["dy"] = normal(case["tokens"], case["hidden"], std=1e-2)
    elif kind == "gemm":
        s["x"], s["w"] = normal(case["m"], case["k"]), normal(case["n"], case["k"], std=case["k"] ** -0.5)
        s["epilogue"] = "silu" if case["silu"] else "none"
    elif kind == "loss":
        s["vocab"] = case["vocab"]
        width = (case["vocab"] + 63) // 64 * 64 if case["padded"] else case["vocab"]
        s["logits"] = normal(case["rows"], width, std=2.0).requires_grad_(True)
        s["targets"] = torch.randint(0, case["vocab"], (case["rows"],), device="cuda", generator=gen)
    elif kind == "norm":
        s["layer"] = FusedLayerNorm(case["d"]).to(device="cuda", dtype=torch.bfloat16)
        with torch.no_grad():
            s["layer"].weight.copy_(normal(case["d"], std=0.2, mean=1.0))
            s["layer"].bias.copy_(normal(case["d"], std=0.1))
        s["x"] = normal(case["rows"], case["d"], std=2.0, mean=0.3).requires_grad_(True)
        s["dy"] = normal(case["rows"], case["d"], std=1e-2)
    elif kind == "optim":
        n = case["elems"]
        s["master"] = torch.randn(n, device="cuda", generator=gen) * 0.02
        s["param"] = s["master"].to(torch.bfloat16)
        s["grad"] = normal(n, std=1e-3)
        s["m"] = torch.randn(n, device="cuda", generator=gen) * 1e-4
        s["v"] = torch.rand(n, device="cuda", generator=gen) * 1e-6
        s["norm_sq"] = torch.zeros(1, device="cuda")
        s["scratch"] = torch.zeros(scratch_floats(n), device="cuda")
        s["clip"] = case["clip"]
    else:
        dt = DTYPES[case["dtype"]]
        x = torch.randn(case["elems"], device="cuda", generator=gen) * 1000
        s["comm"], s["op"], s["x"] = _one_rank(), case["op"], x.to(dt)
        s["out"] = [torch.empty_like(s["x"]) for _ in range(3)]
    return s


# ---- one pass -------------------------------------------------------------------------------------------------------
def run(s):
    kind = s["kind"]
    if kind == "step":
        ddp = s["ddp"]
        if s["replay"] is not None:
            loss = s["replay"](s["idx"], s["targets"])
        else:
            loss = ddp(s["idx"], s["targets"])
            loss.backward()
            ddp.step(lr=3e-4, max_grad_norm=1.0)
        return [loss.detach()] + [b.param for b in ddp.buckets] + [b.exp_avg for b in ddp.buckets]
    if kind == "logits":
        with torch.no_grad():
            return s["model"](s["idx"])
    if kind == "llama":
        model = s["model"]
        model.zero_grad(set_to_none=True)
        loss = model(s["idx"], s["targets"])
        loss.backward()
        return [loss.detach()] + [p.grad for p in model.parameters()]
    if kind in ("mlp", "moe", "norm"):
        y = s["layer"](s["x"])
        return [y.detach(), *torch.autograd.grad(y, [s["x"], *s["layer"].parameters()], s["dy"])]
    if kind == "gemm":
        return gemm(s["x"], s["w"], epilogue=s["epilogue"])
    if kind == "loss":
        # The gradient is written over the logits (that is this entry point's contract), so the next pass on the same
        # state reads those values as its logits: the same work on other numbers.
        loss = fused_cross_entropy(s["logits"], s["targets"], s["vocab"])
        return [loss.detach(), *torch.autograd.grad(loss, [s["logits"]])]
    if kind == "optim":
        sum_squares_(s["grad"], s["norm_sq"], s["scratch"])
        fused_adamw_(s["param"], s["master"], s["m"], s["v"], s["grad"], lr=3e-4, weight_decay=0.1, step=10, zero_grad=False,
                     norm_sq=s["norm_sq"] if s["clip"] else None, max_norm=1.0 if s["clip"] else 0.0)
        return [s["param"], s["master"], s["m"], s["v"], s["norm_sq"]]
    s["comm"].all_reduce(s["x"], s["out"][0], op=s["op"])
    s["comm"].reduce_scatter(s["x"], s["out"][1], op=s["op"])
    s["comm"].all_gather(s["x"], s["out"][2])
    return s["out"]


# ---- what a pass cannot do without ----------------------------------------------------------------------------------
def work(case):
    kind = case["kind"]
    if kind in ("step", "logits", "llama"):
        d, tokens = case["d_model"], case["batch"] * case["seq"]
        per_layer = (4 * d + (3 if kind == "llama" else 2) * case["ffn"]) * d
        matrices = case["layers"] * per_layer + case["vocab"] * d
        attention = 2 * case["layers"] * case["batch"] * case["seq"] ** 2 * d      # causal: half of both products
        if kind == "logits":
            return {"bytes": 2 * (matrices + case["seq"] * d) + 2 * tokens * case["vocab"], "flops": 2 * matrices * tokens + attention}
        flops = 6 * matrices * tokens + 3.5 * attention
        if kind == "llama":
            return {"bytes": 4 * (matrices + case["vocab"] * d), "flops": flops}
        # bf16 weights, fp32 master weights and two fp32 moments: read and written
        return {"bytes": 28 * (matrices + case["seq"] * d), "flops": flops}
    if kind == "mlp":
        t, h, f = case["tokens"], case["hidden"], case["ffn"]
        return {"bytes": 2 * (4 * t * h + 4 * h * f), "flops": 12 * t * h * f}
    if kind == "moe":
        t, h, f, e = case["tokens"], case["hidden"], case["ffn"], case["experts"]
        return {"bytes": 2 * (4 * t * h + 4 * e * h * f), "flops": 12 * t * h * f + 6 * t * h * e}
    if kind == "gemm":
        m, n, k = case["m"], case["n"], case["k"]
        return {"bytes": 2 * (m * k + n * k + m * n), "flops": 2 * m * n * k}
    if kind == "loss":
        return {"bytes": 6 * case["rows"] * case["vocab"], "flops": 8 * case["rows"] * case["vocab"]}
    if kind == "norm":
        # forward reads x, writes y; backward reads x and dy, writes dx
        return {"bytes": 10 * case["rows"] * case["d"], "flops": 20 * case["rows"] * case["d"]}
    if kind == "optim":
        return {"bytes": case["elems"] * (2 + 2 + 24), "flops": 16 * case["elems"]}
    return {"bytes": 3 * 2 * case["elems"] * torch.empty((), dtype=DTYPES[case["dtype"]]).element_size(), "flops": 0}


def tolerance(case):
    kind = case["kind"]
    if kind == "collective":
        return "exact"
    if kind in ("step", "llama"):
        return {"rel": 2e-2}          # bf16 activations and gradients through every layer, forward and backward
    if kind in ("logits", "mlp", "moe"):
        return {"rel": 1e-2}          # a few bf16 roundings in a row
    if kind == "optim":
        return {"rel": 1e-4, "max": 1e-2}       # fp32 sums; a last-bit difference can move a bf16 weight by one of its steps
    return {"rel": 4e-3}              # one bf16 rounding (relative step 2^-8)
