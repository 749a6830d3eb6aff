"""Workloads whose speed is tracked: what a user of the package runs on one GPU, through its public entry points.

Six kinds of work:

* ``train``    one complete step of the Llama trainer (forward, backward, gradient clipping, AdamW);
* ``loss``     evaluation: the mean token loss without gradients;
* ``prefill``  inference over a prompt: the logits that follow its last token;
* ``attention``  the attention kernels by themselves, forward and backward, on a packed QKV activation;
* ``encode``   a list of gradients packed into one fp8 buffer and unpacked again, as a quantised collective does;
* ``outer``    the outer optimizer step of DiLoCo on one fragment.

The sizes come from the model configurations of :mod:`torchft_b200.models.llama`, the benchmarks (``bench.py``: sequence
8192, one sequence per GPU; ``bench_diloco.py``: sequence 2048, the 1B model in four fragments) and the examples.  The
8B model's training state does not fit a GPU next to other states, so its cases keep the model's widths and
vocabulary and take 4 of its 32 layers; the 1B model trains with 4 of its 16 because the rounding noise of bf16
gradients grows with depth, and with it what two correct implementations differ by.
"""

import dataclasses
import math

import torch
from torch import nn

from torchft_b200.models.lenet import LeNet
from torchft_b200.models.llama import CONFIGS
from torchft_b200.ops import kernels as K
from torchft_b200.ops.diloco import outer_step_
from torchft_b200.parallel.hsdp import ShardedLlamaTrainer
from torchft_b200.quantization import fused_dequantize_from_fp8, fused_quantize_into_fp8


def listed():
    return [
        # the smallest training step: examples, CI and debugging runs; launches and host work count, not the chip
        {"name": "train-tiny", "kind": "train", "model": "llama-tiny", "layers": 2, "batch": 1, "seq": 256, "chunks": 4},
        # a small model on documents cut to a length that is no multiple of anything
        {"name": "train-small-ragged", "kind": "train", "model": "llama-small", "layers": 4, "batch": 3, "seq": 1000, "chunks": 4},
        # the inner step of the DiLoCo benchmark: a quarter of the 1B model's layers, head dim 64, sequence 2048
        {"name": "train-1b", "kind": "train", "model": "llama3-1b", "layers": 4, "batch": 4, "seq": 2048, "chunks": 1},
        # the headline benchmark's step: 8B widths, head dim 128, one sequence of 8192
        {"name": "train-8b-width", "kind": "train", "model": "llama3-8b", "layers": 4, "batch": 1, "seq": 8192, "chunks": 1},
        # evaluation of a 1B model on a few sequences between training steps
        {"name": "loss-1b", "kind": "loss", "model": "llama3-1b", "layers": 16, "batch": 2, "seq": 2048, "chunks": 4},
        # a prompt of ordinary length through 8B-width layers
        {"name": "prefill-8b-width", "kind": "prefill", "model": "llama3-8b", "layers": 4, "batch": 1, "seq": 1536, "chunks": 4},
        # attention of the 8B model at the benchmark's sequence length
        {"name": "attention-128", "kind": "attention", "batch": 1, "seq": 8192, "heads": 32, "kv_heads": 8, "head_dim": 128, "causal": True},
        # attention of the 1B model at the DiLoCo benchmark's batch
        {"name": "attention-64", "kind": "attention", "batch": 8, "seq": 2048, "heads": 32, "kv_heads": 8, "head_dim": 64, "causal": True},
        # fp8 exchange of a small model's gradients: ten tensors of odd sizes
        {"name": "encode-lenet", "kind": "encode", "model": "lenet", "layers": 0, "dtype": "float32", "world": 2},
        # fp8 exchange of a quarter of the 1B model: bf16 gradients of four layers, eight groups
        {"name": "encode-1b-quarter", "kind": "encode", "model": "llama3-1b", "layers": 4, "dtype": "bfloat16", "world": 8},
        # outer Nesterov step on the same quarter in fp32 (the trainer's master weights)
        {"name": "outer-1b-quarter", "kind": "outer", "n": 243286016, "dtype": "float32", "alpha": 0.5},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_engine(rng, kind):
    model = rng.choice(["llama-tiny", "llama-small", "llama3-1b", "llama3-8b"])
    top = {"llama-tiny": 16384, "llama-small": 16384, "llama3-1b": 8192, "llama3-8b": 8192}[model]
    layers = rng.randint(1, {"llama-tiny": 4, "llama-small": 8, "llama3-1b": 4, "llama3-8b": 4}[model])
    seq = _log_int(rng, 64, min(top, 8192))
    if rng.random() < 0.7:  # most jobs pack their sequences to a round length
        seq = max(256, seq // 256 * 256)
    batch = max(1, min(16, _log_int(rng, 1, max(1, top // seq))))
    return {"kind": kind, "model": model, "layers": layers, "batch": batch, "seq": seq, "chunks": rng.choice([1, 4])}


def draw(rng):
    """One more case of the same ranges."""
    kind = rng.choice(["train", "train", "train", "loss", "prefill", "attention", "attention", "encode", "outer"])
    if kind in ("train", "loss", "prefill"):
        return _draw_engine(rng, kind)
    if kind == "attention":
        head_dim = rng.choice([64, 128])
        step = 256 if head_dim == 64 else 128
        seq = max(step, _log_int(rng, 128, 8192) // step * step)
        kv_heads = rng.choice([1, 2, 4, 8])
        return {"kind": kind, "batch": _log_int(rng, 1, max(1, 16384 // seq)), "seq": seq,
                "heads": kv_heads * rng.choice([1, 2, 4]), "kv_heads": kv_heads, "head_dim": head_dim,
                "causal": rng.random() < 0.8}
    if kind == "encode":
        model = rng.choice(["lenet", "llama-tiny", "llama-small", "llama3-1b"])
        return {"kind": kind, "model": model, "layers": rng.randint(1, 4), "dtype": rng.choice(["bfloat16", "float32"]),
                "world": rng.choice([2, 3, 4, 8])}
    n = _log_int(rng, 1 << 12, 1 << 28)
    return {"kind": kind, "n": n - n % 4, "dtype": rng.choice(["float32", "float32", "bfloat16"]),
            "alpha": rng.choice([0.0, 0.5])}


# ---------------------------------------------------------------------------------------------------------------------


def _config(case):
    return dataclasses.replace(CONFIGS[case["model"]], n_layers=case["layers"])


def _gradient_shapes(case):
    if case["model"] == "lenet":
        return [tuple(p.shape) for p in LeNet().parameters()]
    cfg = _config(case)
    return [shape for u in range(1, cfg.n_layers + 1) for _, shape in cfg.unit_fields(u)]


def prepare(case, seed):
    device = torch.device("cuda", torch.cuda.current_device())
    g = torch.Generator(device=device)
    g.manual_seed(seed)
    kind = case["kind"]
    if kind in ("train", "loss", "prefill"):
        # random-init weights and uniform token ids, as the benchmarks use them; a learning rate from a job's warm-up
        cfg = _config(case)
        trainer = ShardedLlamaTrainer(cfg, case["batch"], case["seq"], device, lr=1e-5, seed=seed % 1000003,
                                      logit_chunks=case["chunks"])
        tok = torch.randint(0, cfg.vocab_size, (case["batch"], case["seq"] + 1), generator=g, device=device)
        return {"kind": kind, "trainer": trainer, "tokens": tok[:, :-1].contiguous(), "targets": tok[:, 1:].contiguous()}
    if kind == "attention":
        B, S, H, Hk, D = (case[k] for k in ("batch", "seq", "heads", "kv_heads", "head_dim"))
        bf = dict(dtype=torch.bfloat16, device=device)
        # q, k and v are column slices of one packed projection; so are their gradients
        qkv = torch.randn(B * S, (H + 2 * Hk) * D, generator=g, **bf)
        return {"kind": kind, "shape": (B, S, H, Hk, D), "causal": case["causal"], "qkv": qkv, "dqkv": torch.empty_like(qkv),
                "out": torch.empty(B * S, H * D, **bf), "d_out": torch.randn(B * S, H * D, generator=g, **bf),
                "lse": torch.empty(B, H, S, dtype=torch.float32, device=device)}
    dtype = getattr(torch, case["dtype"])
    if kind == "encode":
        # gradients: normal, each tensor with a magnitude of its own
        grads = [torch.randn(s, generator=g, device=device, dtype=dtype).mul_(1e-3 * (1 + i % 7)) for i, s in enumerate(_gradient_shapes(case))]
        return {"kind": kind, "grads": grads, "back": [torch.empty_like(t) for t in grads], "world": case["world"]}
    n = case["n"]

    def normal(std, dt):
        return torch.randn(n, generator=g, device=device, dtype=dt).mul_(std)

    return {"kind": kind, "alpha": case["alpha"], "g": normal(1e-3, dtype), "momentum": normal(1e-3, torch.float32),
            "backup": normal(0.02, dtype), "param": normal(0.02, dtype)}


def run(state):
    kind = state["kind"]
    if kind == "train":
        tr = state["trainer"]
        loss = tr.train_step(state["tokens"], state["targets"])
        return {"loss": loss, "grad_norm": tr.grad_norm, "grads": tr.g_flat, "weights": tr.p_flat, "master": tr.master_flat, "m": tr.m_flat}
    if kind == "loss":
        eng = state["trainer"].engine
        return {"loss": eng.forward(state["tokens"], state["targets"], train=False), "rows": eng.loss_rows}
    if kind == "prefill":
        return state["trainer"].engine.forward(state["tokens"], None, train=False)
    if kind == "attention":
        B, S, H, Hk, D = state["shape"]
        qkv, dqkv, out, lse = state["qkv"], state["dqkv"], state["out"], state["lse"]
        a, b = H * D, (H + Hk) * D
        q, k, v = qkv[:, :a], qkv[:, a:b], qkv[:, b:]
        K.attention_fwd(q, k, v, B, S, H, Hk, D, out, lse, causal=state["causal"])
        K.attention_bwd(q, k, v, out, state["d_out"], lse, dqkv[:, :a], dqkv[:, a:b], dqkv[:, b:], B, S, H, Hk, D,
                        causal=state["causal"])
        return {"out": out, "lse": lse, "dqkv": dqkv}
    if kind == "encode":
        buf, sizes = fused_quantize_into_fp8(state["grads"], state["world"])
        fused_dequantize_from_fp8(state["back"], buf, state["world"])
        return {"buf": buf, "n": sizes[0], "back": state["back"]}
    outer_step_(state["g"], state["momentum"], state["backup"], state["param"], 0.7, 0.9, state["alpha"])
    return {"momentum": state["momentum"], "backup": state["backup"], "param": state["param"]}


def work(case):
    kind = case["kind"]
    if kind in ("train", "loss", "prefill"):
        cfg = _config(case)
        tokens = case["batch"] * case["seq"]
        params = cfg.num_params()
        flops = cfg.flops_per_token(case["seq"]) * tokens
        if kind == "train":
            # weights in bf16, master weights and two moments in fp32, read and written; gradients written
            return {"bytes": params * (2 * (2 + 12) + 2) + tokens * 16, "flops": flops}
        head = 2.0 * cfg.vocab_size * cfg.dim * tokens
        if kind == "loss":
            return {"bytes": params * 2 + tokens * 20, "flops": flops / 3}
        return {"bytes": params * 2 + tokens * 8 + cfg.vocab_size * 2, "flops": flops / 3 - head + head / tokens}
    if kind == "attention":
        B, S, H, Hk, D = (case[k] for k in ("batch", "seq", "heads", "kv_heads", "head_dim"))
        pairs = B * H * (S * (S + 1) / 2 if case["causal"] else float(S) * S)
        # forward two products, backward five; q, k, v, dO read, O, dq, dk, dv written
        return {"bytes": B * S * (2 * (H + 2 * Hk) * D * 2 + 2 * H * D * 2 + H * 4), "flops": 7 * 2.0 * pairs * D}
    size = 2 if case["dtype"] == "bfloat16" else 4
    if kind == "encode":
        n = sum(math.prod(s) for s in _gradient_shapes(case))
        return {"bytes": n * (2 * size + 2 * (1 + 4 / 128)), "flops": 0}
    return {"bytes": case["n"] * (5 * size + 2 * 4), "flops": 0}


def tolerance(case):
    kind = case["kind"]
    if kind == "train":
        # Gradients of a freshly initialised decoder carry the bf16 rounding of every activation before them.  With
        # the library's attention and the one-CTA GEMM in place of the default kernels they move by 0.6 % (tiny) to
        # 1.7 % (8B widths, four layers) in norm.
        return {"rel": 0.03}
    if kind == "loss":
        return {"rel": 0.008}  # 0.2 % between the same two sets of kernels
    if kind == "prefill":
        return {"rel": 0.03}  # 1.2 %
    if kind == "attention":
        return {"rel": 0.012}  # 0.25 % from an fp32 evaluation of the same bf16 inputs, for every output
    if kind == "encode":
        return "exact"
    return {"rel": 1e-5 if case["dtype"] == "float32" else 2e-3}  # one rounding per element
