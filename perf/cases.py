"""The calls of this framework whose speed its users feel, as plain cases.

A user of this package trains Llama models: the fused engine's ``train_step`` from the two-block debug models up to the
blocks of the 10B production model, with and without packed documents, gradient accumulation, activation checkpointing,
z-loss and fp32 gradient reduction. Around it stand the forward-only pass (evaluation), the autograd module with the
fused head and loss (users who bring their own optimizer), and the uint8 quantiser of the DiLoCo pseudo-gradient.

``listed()`` are the fixed cases, ``draw()`` gives others from the same ranges, ``prepare()`` builds what a training
program holds before the call, ``run()`` is one call through the public entry points.
"""
from __future__ import annotations

import math
import random
from dataclasses import replace

import torch

from prime_b200.engine.fused_llama import FusedLlama
from prime_b200.loss import compute_cross_entropy_loss
from prime_b200.models.llama import Transformer, bench_configs, llama2_configs, llama3_configs
from prime_b200.ops import kernels as K
from prime_b200.ops import quant

# Presets with their vocabularies: those of the tokenizers that the configurations name (32000 words for the llama2
# family, 128256 for llama3) and the 1024 ids of the fake-data debug runs.
_MODELS = {
    "tiny": bench_configs["tiny"],
    "debug2": replace(llama2_configs["debugmodel"], vocab_size=1024),       # head size 32
    "debug3": replace(llama3_configs["debugmodel"], vocab_size=1024),       # head size 16
    "70M": replace(llama2_configs["70M"], vocab_size=32000),
    "150M": bench_configs["150M"],
    "271M": replace(llama2_configs["271M"], vocab_size=32000),              # head size 128
    "1B": bench_configs["1B"],
    "10B": bench_configs["10B"],                                            # GQA 32 / 8 heads of 128, 128256 words
}
_Z = {"none": K.Z_NONE, "max": K.Z_MAX, "lse": K.Z_LSE}


def _step(name, model, batch, seq, micro=0, packed=False, z="none", ac=False, fp32_grads=False, layers=0):
    return {"name": name, "kind": "step", "model": model, "layers": layers, "batch": batch, "seq": seq, "micro": micro or batch,
            "packed": packed, "z": z, "ac": ac, "fp32_grads": fp32_grads}


def listed():
    return [
        # smallest useful step (the two-block model of the tiny configuration, 512 tokens): launches and latency count
        _step("step_tiny", "tiny", 4, 128),
        # configs/debug/normal.toml as it stands: fake data, 16 sequences in micro-batches of 8, heads of 32 columns
        _step("step_debug", "debug2", 16, 1024, micro=8),
        # 70M on tokenised text: documents packed into rows, two micro-batches, gradients reduced in fp32
        _step("step_70M_packed", "70M", 32, 1024, micro=16, packed=True, fp32_grads=True),
        # the headline benchmark: 150M, 64 x 1024 tokens in one micro-batch
        _step("step_150M", "150M", 64, 1024),
        # the 1B model of the DiLoCo benchmark at its 2048-token rows
        _step("step_1B", "1B", 8, 2048),
        # four of the 42 blocks of the 10B production run (configs/10B): one packed 8192-token row, activation
        # checkpointing, max z-loss; fp32 gradients, since frequent words add up hundreds of rows in the embedding's
        _step("step_10B_4blocks", "10B", 1, 8192, packed=True, z="max", ac=True, fp32_grads=True, layers=4),
        # evaluation of a handful of ragged prompts: forward only, sizes that divide nothing
        {"name": "logits_150M_ragged", "kind": "logits", "model": "150M", "layers": 0, "batch": 3, "seq": 777, "packed": False},
        # evaluation of the 1B model on full rows of packed documents
        {"name": "logits_1B", "kind": "logits", "model": "1B", "layers": 0, "batch": 4, "seq": 2048, "packed": True},
        # the autograd module with the fused head and loss: fp32 parameters, forward and backward
        {"name": "module_70M", "kind": "module", "model": "70M", "batch": 8, "seq": 1024, "packed": False, "z": "lse"},
        # uint8 quantisation of one worker's pseudo-gradient: the 150M model on one GPU
        {"name": "quantize_150M", "kind": "quantize", "n": _MODELS["150M"].num_params()},
    ]


def _log_int(rng: random.Random, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random):
    kind = rng.choice(["step", "step", "step", "step", "logits", "module", "quantize"])
    if kind == "quantize":
        return {"kind": kind, "n": _log_int(rng, 4096, 1 << 28)}
    packed = rng.random() < 0.5
    if kind == "module":
        model = rng.choice(["debug2", "debug3", "70M"])
        tokens = _log_int(rng, 512, 16384)
        seq = min(_log_int(rng, 64, 4096), tokens)
        return {"kind": kind, "model": model, "batch": max(1, tokens // seq), "seq": seq, "packed": packed,
                "z": rng.choice(["none", "lse"])}
    if kind == "logits":
        model = rng.choice(["tiny", "70M", "150M", "271M", "1B"])
        tokens = _log_int(rng, 64, 8192)
        seq = min(_log_int(rng, 32, 8192), tokens)
        return {"kind": kind, "model": model, "layers": 0, "batch": max(1, tokens // seq), "seq": seq, "packed": packed}
    model = rng.choice(["tiny", "debug2", "debug3", "70M", "150M", "271M", "1B", "10B"])
    cap = {"10B": 8192, "1B": 16384, "271M": 32768}.get(model, 65536)
    tokens = _log_int(rng, 512, cap)
    seq = min(_log_int(rng, 64, 8192), tokens)
    batch = max(1, tokens // seq)
    micro = batch
    if batch % 2 == 0 and rng.random() < 0.4:
        micro = batch // 2
    c = _step("", model, batch, seq, micro=micro, packed=packed, z=rng.choice(["none", "none", "max", "lse"]),
              ac=model == "10B" or rng.random() < 0.2, fp32_grads=packed if model == "10B" else rng.random() < 0.25,
              layers=rng.choice([1, 2, 3]) if model == "10B" else 0)
    del c["name"]
    return c


# ------------------------------------------------------------------------------------------------ inputs
def _args(case):
    a = _MODELS[case["model"]]
    return replace(a, max_seq_len=max(case["seq"], 64), n_layers=case.get("layers") or a.n_layers, init_mode="reference",
                   fused_linear_ce=case["kind"] == "module")


def _doc_lengths(case, seed: int) -> list[list[int]]:
    """Document lengths of every packed row: log-uniform from 16 tokens to a whole row, cut at the row's end."""
    rng = random.Random(seed)
    rows = []
    for _ in range(case["batch"]):
        left, row = case["seq"], []
        while left:
            n = min(left, _log_int(rng, min(16, case["seq"]), case["seq"]))
            row.append(n)
            left -= n
        rows.append(row)
    return rows


def _batch(case, args, seed: int):
    """Token ids, next-token labels and the document map. Packed text has word frequencies of about 1 / rank; the
    unpacked cases use uniform ids like the fake-data loader."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    B, T, V = case["batch"], case["seq"], args.vocab_size
    if case["packed"]:
        u = torch.rand(B, T + 1, device="cuda", generator=g)
        rank = (torch.exp(u * math.log(V)) - 1.0).long().clamp_(0, V - 1)
        ids = torch.randperm(V, device="cuda", generator=g)[rank]
        starts = []
        for b, row in enumerate(_doc_lengths(case, seed)):
            pos = b * T
            for n in row:
                starts += [pos] * n
                pos += n
        seq_start = torch.tensor(starts, dtype=torch.int32).cuda()
    else:
        ids = torch.randint(0, V, (B, T + 1), device="cuda", generator=g)
        seq_start = None
    return ids[:, :-1].contiguous(), ids[:, 1:].contiguous(), seq_start


def prepare(case, seed: int):
    """Inputs made from ``seed`` and the engine, module or buffer that the program keeps between calls."""
    if case["kind"] == "quantize":
        # pseudo-gradient of 100 inner AdamW steps: bell-shaped with a few heavy rows
        g = torch.Generator(device="cuda").manual_seed(seed)
        x = torch.randn(case["n"], device="cuda", generator=g).mul_(1e-3)
        x[: case["n"] // 64].mul_(8.0)
        return {"case": case, "x": x}
    args = _args(case)
    tokens, labels, seq_start = _batch(case, args, seed)
    st = {"case": case, "tokens": tokens, "labels": labels, "seq_start": seq_start}
    torch.manual_seed(seed)
    with torch.device("cuda"):
        model = Transformer(args)               # the presets' own initialisation, as training starts from it
    if case["kind"] == "module":
        st["model"] = model
        return st
    eng = FusedLlama(args, device="cuda", z_mode=_Z[case.get("z", "none")], z_weight=2e-4 if case.get("z", "none") != "none" else 0.0,
                     ac_ckpt=case.get("ac", False), grad_dtype=torch.float32 if case.get("fp32_grads") else torch.bfloat16)
    eng.load_from_module(model)
    st["engine"] = eng
    return st


# ------------------------------------------------------------------------------------------------ one pass
def run(state):
    """One optimizer step, forward pass, forward and backward, or quantisation; returns everything it produced."""
    case = state["case"]
    if case["kind"] == "quantize":
        q, lut = quant.uniform_8bit_quantize_cuda(state["x"])
        return {"q": q, "codebooks": lut}
    if case["kind"] == "logits":
        return {"logits": state["engine"].forward_logits(state["tokens"], seq_start=state["seq_start"])}
    if case["kind"] == "module":
        model = state["model"]
        model.zero_grad(set_to_none=True)
        h = model(state["tokens"], seq_start=state["seq_start"])
        ce, z = compute_cross_entropy_loss(h, state["labels"], z_weight=2e-4 if case["z"] == "lse" else None,
                                           fused_linear_weight=model.output.weight)
        (ce if z is None else ce + z).backward()
        return {"loss": ce.detach(), "grads": [p.grad for p in model.parameters()]}
    eng = state["engine"]
    loss, norm = eng.train_step(state["tokens"], state["labels"], lr=4e-5, micro_bs=case["micro"], seq_start=state["seq_start"])
    return {"loss": loss, "grad_norm": norm, "grads": eng.grads, "master": eng.master, "exp_avg": eng.exp_avg,
            "exp_avg_sq": eng.exp_avg_sq, "params": eng.params}


# ------------------------------------------------------------------------------------------------ floors
def work(case):
    """Bytes and operations of one pass: inputs once in, outputs once out, no recomputation, visible pairs only."""
    if case["kind"] == "quantize":
        n = case["n"]
        return {"bytes": 5.0 * n + 1024.0 * -(-n // 16384), "flops": 0.0}
    a = _args(case)
    M = case["batch"] * case["seq"]
    pairs = (sum(n * (n + 1) // 2 for row in _doc_lengths(case, 0) for n in row) if case["packed"]
             else case["batch"] * case["seq"] * (case["seq"] + 1) // 2)
    P = a.num_params()
    matmul = P - a.vocab_size * a.dim - (2 * a.n_layers + 1) * a.dim        # without the embedding table and the norms
    attn = 4.0 * a.head_dim * a.n_heads * pairs * a.n_layers                # Q K^T and P V over the visible pairs
    fwd = 2.0 * matmul * M + attn
    if case["kind"] == "logits":
        return {"bytes": 2.0 * P + 8.0 * M + 4.0 * M * a.vocab_size, "flops": fwd}
    if case["kind"] == "module":
        return {"bytes": 8.0 * P + 16.0 * M, "flops": 3.0 * fwd}            # fp32 parameters in, fp32 gradients out
    grad = 4.0 if case["fp32_grads"] else 2.0
    # bf16 parameters in and out, gradients out, fp32 master weights and both moments in and out
    return {"bytes": (4.0 + grad + 24.0) * P + 16.0 * M, "flops": 3.0 * fwd}


def tolerance(case):
    if case["kind"] == "quantize":
        # bytes are whole numbers of a fixed rounding rule; a value within one fp32 rounding of a bin's edge may go either way
        return {"rel": 1e-5, "max": 1e-3, "differ": 1e-5}
    # bf16 activations: the same network with its GEMM tiles summed in another order moves gradients by 0.1-0.25 % up to
    # eight blocks of 512 columns, by 0.6-0.9 % (second moments 1.1 %) at the 12 to 18 blocks of the larger models, logits by
    # 0.3-0.7 %. Single values move by more where a sum cancels.
    deep = case["model"] in ("150M", "271M", "1B", "10B")
    return {"rel": 3e-2 if deep else 1e-2, "max": 0.99}
