"""Workloads of the framework on one GPU, as its users run them: training steps, gradients for test-time training, scoring,
logits and GPTQ export. `listed()` names the standing cases, `draw(rng)` gives further ones of the same ranges, `prepare` builds
what a program holds before the call, `run` is one call through the public entry points, `work` what it cannot do without and
`tolerance` how far two correct implementations at the same precision may differ.

Model shapes are the framework's own families (`family_preset`); token streams are the seeded Zipf / Markov tokens of the
synthetic shards; weights and optimizer state have the distributions of a run in progress (dense projections, non-trivial
controls, a filled momentum), so that every output is determined by the inputs and not by rounding noise around zero."""
import math

import numpy as np
import torch

from parameter_golf_b200.data.bpb import BpbLuts
from parameter_golf_b200.data.shards import generate_markov_tokens
from parameter_golf_b200.eval.sliding import eval_sliding
from parameter_golf_b200.eval.ttt import init_q_lora
from parameter_golf_b200.models import gpt
from parameter_golf_b200.models.engine import EngineBackend, EngineRunner
from parameter_golf_b200.quant.gptq import gptq_quantize
from parameter_golf_b200.spec import family_preset

DEVICE = "cuda:0"
FAMILIES = ("record_11l", "baseline_9l", "recurrence_mid_sp8192")


def listed():
    return [
        # One evaluation window scored by itself: the shortest call of the scoring path (a sequence handed over one at a time).
        {"name": "score_1x2048", "kind": "score", "family": "record_11l", "batch": 1, "seq": 2048},
        # The final evaluation of a run: sliding windows of 2048 tokens at stride 64 in batches of 32 windows, from host tokens to
        # (loss, bits per byte), over three batches (the last one ragged).
        {"name": "sliding_85_windows", "kind": "sliding", "family": "record_11l", "tokens": 85 * 64, "window": 2048, "stride": 64, "batch": 32},
        # Soft-capped logits over the 8192-token vocabulary of the sweep families for an odd batch of part-length sequences.
        {"name": "logits_5x896_sp8192", "kind": "logits", "family": "recurrence_mid_sp8192", "batch": 5, "seq": 896},
        # Test-time training on a ragged rest of a chunk: forward and backward of a few sequences, gradients of every parameter.
        {"name": "adapt_3x1920", "kind": "adapt", "family": "record_11l", "batch": 3, "seq": 1920},
        # Test-time training at its full batch of 32 sequences (one chunk of 65,536 tokens).
        {"name": "adapt_32x2048", "kind": "adapt", "family": "record_11l", "batch": 32, "seq": 2048},
        # Phased LoRA test-time training of an 8192-token family: adapter of rank 128 on the queries, adapter gradients only.
        {"name": "adapt_lora_12x2048_sp8192", "kind": "lora", "family": "recurrence_mid_sp8192", "batch": 12, "seq": 2048, "rank": 128},
        # Optimizer steps through the trainer's own call (page-locked token spans in, mean loss and updated weights out).
        # A smoke-mode step: two sequences, where launches and latency count.
        {"name": "train_record_4k", "kind": "train", "family": "record_11l", "tokens": 2 * 2048, "seq": 2048, "accum": 1, "option": "default"},
        # One rank's share of the record step on eight GPUs: one micro-batch of 48 x 2048 tokens and the whole optimizer step.
        {"name": "train_record_98k", "kind": "train", "family": "record_11l", "tokens": 48 * 2048, "seq": 2048, "accum": 1, "option": "default"},
        # The headline workload: the record step on one GPU, 8 micro-batches of 48 x 2048 tokens.
        {"name": "train_record_786k", "kind": "train", "family": "record_11l", "tokens": 384 * 2048, "seq": 2048, "accum": 8, "option": "default"},
        # The baseline trainer's step on one GPU: 524,288 tokens in sequences of 1024, relu^2, full rotary embedding.
        {"name": "train_baseline_524k", "kind": "train", "family": "baseline_9l", "tokens": 512 * 1024, "seq": 1024, "accum": 8, "option": "default"},
        # A proxy-mode step of an 8192-token family: recurrent blocks, value embeddings, boundary-masked smear gate.
        {"name": "train_sp8192_16k", "kind": "train", "family": "recurrence_mid_sp8192", "tokens": 8 * 2048, "seq": 2048, "accum": 1, "option": "default"},
        # Export: full-Hessian GPTQ of one block's MLP down projection (512 x 1536), five clip candidates.
        {"name": "gptq_512x1536", "kind": "gptq", "rows": 512, "cols": 1536, "bits": 6},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("score", "score", "sliding", "logits", "adapt", "adapt", "lora", "train", "train", "train", "train", "gptq"))
    fam = rng.choice(FAMILIES)
    if kind == "gptq":
        return {"kind": kind, "rows": _log_int(rng, 48, 768), "cols": 8 * _log_int(rng, 32, 192), "bits": rng.choice((5, 6, 8))}
    if kind == "sliding":
        return {"kind": kind, "family": "record_11l", "tokens": _log_int(rng, 700, 12000), "window": 128 * rng.randint(4, 16), "stride": 64, "batch": rng.choice((16, 32))}
    seq = 128 * _log_int(rng, 4, 32)                     # 512 .. 4096
    if kind in ("score", "logits"):
        most = (65536 if kind == "score" else 16384) // seq
        return {"kind": kind, "family": fam, "batch": _log_int(rng, 1, most), "seq": seq}
    if kind == "adapt":
        return {"kind": kind, "family": fam, "batch": _log_int(rng, 1, 65536 // seq), "seq": seq}
    if kind == "lora":
        return {"kind": kind, "family": fam, "batch": _log_int(rng, 1, 32768 // seq), "seq": seq, "rank": rng.choice((8, 16, 80, 128))}
    option = rng.choice(("default", "default", "default", "default", "cuda_graph", "reproducible", "recompute"))
    accum = rng.choice((1, 1, 2))
    return {"kind": kind, "family": fam, "tokens": seq * accum * _log_int(rng, 1, 98304 // seq), "seq": seq, "accum": accum, "option": option}


# ---- what a program holds before the call ---------------------------------------------------------------------------------

def _spec(case):
    spec = family_preset(case["family"])
    m, t = spec.model, spec.train
    if m.bigram.enabled and m.bigram.dim % 64:
        m.bigram.dim = 128                               # the CUDA backends take tables in multiples of 64 columns
    t.backend, t.world_size, t.rank = "cuda_single", 1, 0
    t.distributed_optimizer_backend = "all_reduce_replicated_muon"
    t.max_wallclock_seconds = 0.0
    if case["kind"] == "train":
        spec.mode = "record_shaped_proxy"
        t.seq_len, t.batch_tokens, t.grad_accum_steps = case["seq"], case["tokens"], case["accum"]
        m.train_seq_len = case["seq"]
        t.cuda_graph = case["option"] == "cuda_graph"
        t.reproducible_backward = case["option"] == "reproducible"
        t.save_layer_acts = "none" if case["option"] == "recompute" else "all"
    elif case["kind"] == "sliding":
        m.eval_seq_len = case["window"]
    return spec.validate()


def _weights(m, gen):
    """Weights as a run in progress has them: projections of unit gain, controls around their working points."""
    p = {}
    for name, shape in gpt.param_shapes(m).items():
        x = torch.randn(shape, generator=gen, device=DEVICE)
        if name in gpt.BANKS:
            x *= shape[-1] ** -0.5
        elif name in ("tok_emb", "bigram_embed", "ve_embed"):
            x *= 0.05
        elif name in ("bigram_proj", "ve_proj"):
            x *= shape[-1] ** -0.5
        elif name in ("attn_scale", "mlp_scale"):
            x = 0.3 + 0.05 * x
        elif name == "resid_mix":
            x *= 0.1
            x[:, 0] += 0.9
        elif name == "q_gain":
            x = 1.5 * (1.0 + 0.1 * x)
        elif name == "skip_weights":
            x = 0.7 + 0.1 * x
        elif name in ("bigram_scale", "ve_scale"):
            x = torch.full(shape, 0.3, device=DEVICE)
        elif name == "ve_layer_scales":
            x = 1.0 + 0.1 * x
        p[name] = x
    return p


def _tokens(count, vocab, seed):
    return generate_markov_tokens(count, vocab, seed=1000003 * (seed + 1), chain_seed=7)


def _batch(case, vocab, seed):
    b, s = case["batch"], case["seq"]
    span = torch.from_numpy(_tokens(b * s + 1, vocab, seed).astype(np.int64)).to(DEVICE)
    return span[:-1].reshape(b, s).contiguous(), span[1:].reshape(b, s).contiguous()


def prepare(case, seed):
    kind = case["kind"]
    gen = torch.Generator(device=DEVICE).manual_seed(7919 * seed + 13)
    if kind == "gptq":
        rows, cols = case["rows"], case["cols"]
        x = torch.randn(2 * cols, cols, generator=gen, device=DEVICE) * torch.linspace(0.3, 2.0, cols, device=DEVICE)
        x = x + 0.5 * x.roll(1, dims=1)                  # correlated inputs with unequal powers
        w = torch.randn(rows, cols, generator=gen, device=DEVICE) * cols ** -0.5
        return {"kind": kind, "W": w, "H": x.t() @ x / x.shape[0], "bits": case["bits"]}
    spec = _spec(case)
    m = spec.model
    params = _weights(m, gen)
    if kind == "train":
        backend = EngineBackend(spec, params)
        e = backend.engine
        # optimizer state of a run in progress
        backend.load_state_dict({
            "mom": {k: 1e-3 * torch.randn(params[k].shape, generator=gen, device=DEVICE) for k in gpt.BANKS}, "adam_t": 1000,
            "m": [1e-4 * torch.randn(g["m"].shape, generator=gen, device=DEVICE) for g in e.groups],
            "v": [torch.full_like(g["v"], 4e-8) for g in e.groups],
            "ema_banks": {k: params[k] for k in gpt.BANKS}, "ema_groups": [g["p"].clone() for g in e.groups]})
        n = case["tokens"] // case["accum"]
        toks = _tokens(case["accum"] * n + 1, m.vocab_size, seed)
        spans = backend.host_spans(case["accum"])
        for i, s in enumerate(spans):
            s.copy_(torch.from_numpy(toks[i * n:(i + 1) * n + 1].view(np.int16)))
        return {"kind": kind, "backend": backend, "spans": spans}
    runner = EngineRunner(spec, params, DEVICE)
    if kind == "sliding":
        return {"kind": kind, "runner": runner, "tokens": _tokens(case["tokens"] + 1, m.vocab_size, seed), "window": case["window"],
                "stride": case["stride"], "batch": case["batch"], "luts": BpbLuts.seeded(m.vocab_size, spec.eval.byte_table_seed)}
    if kind == "lora":
        runner.lora = init_q_lora(m, case["rank"], 144.0, DEVICE)
        runner.lora["b"].normal_(0.0, 0.02, generator=gen)
    ids, tgt = _batch(case, m.vocab_size, seed)
    runner.nll(ids, tgt)                                 # the runner lays out its weights and buffers at its first call
    return {"kind": kind, "runner": runner, "ids": ids, "tgt": tgt}


def run(state):
    kind = state["kind"]
    if kind == "gptq":
        return gptq_quantize(state["W"], state["H"], state["bits"])
    if kind == "train":
        backend = state["backend"]
        loss = backend.train_step_spans(state["spans"], 0.1, 0.95)
        return {"loss": loss, **backend.sync_params()}
    r = state["runner"]
    if kind == "sliding":
        return eval_sliding(r.nll, state["tokens"], state["window"], state["stride"], state["luts"], batch_windows=state["batch"], device=DEVICE)
    if kind == "score":
        return r.nll(state["ids"], state["tgt"])
    if kind == "logits":
        return r.logits(state["ids"])
    return r.loss_and_grads(state["ids"], state["tgt"], names=[] if kind == "lora" else None)


# ---- what a pass cannot do without ------------------------------------------------------------------------------------------

def work(case):
    if case["kind"] == "gptq":
        r, c = case["rows"], case["cols"]
        # factorising the Hessian and its inverse, then five candidates of the triangular error feedback
        return {"bytes": 4.0 * (r * c + c * c) + r * (c + 4.0), "flops": 4.0 / 3.0 * c ** 3 + 5.0 * r * c * c}
    spec = _spec(case)
    m = spec.model
    d, blocks = m.model_dim, len(gpt.layer_schedule(m))
    mats = d * (d + 2 * m.kv_dim) + d * d + 2 * d * m.mlp_dim
    params = float(gpt.count_params(m))
    if case["kind"] == "sliding":
        seq = case["window"]
        starts = [ws for ws in range(0, case["tokens"], case["stride"])]
        tokens = float(sum(min(ws + seq, case["tokens"]) - ws for ws in starts))
    elif case["kind"] == "train":
        seq, tokens = case["seq"], float(case["tokens"])
    else:
        seq, tokens = case["seq"], float(case["batch"] * case["seq"])
    fixed = blocks * mats + d * m.vocab_size + (d * m.bigram.dim if m.bigram.enabled else 0)
    if m.value_embedding.enabled:
        fixed += len(m.value_embedding.layers) * m.value_embedding.dim * m.kv_dim
    dense, attn = 2.0 * tokens * fixed, 2.0 * tokens * seq * d * blocks            # causal: half of the square, two products
    kind = case["kind"]
    if kind == "train":
        # fp32 weights, momentum, Adam moments and averages read and written once; tokens in
        state = 4.0 * 2.0 * 3.0 * params
        return {"bytes": state + 2.0 * tokens, "flops": 3.0 * dense + 3.5 * attn}
    if kind == "adapt":
        return {"bytes": 8.0 * params + 16.0 * tokens, "flops": 3.0 * dense + 3.5 * attn}
    if kind == "lora":
        low = 2.0 * tokens * blocks * 2.0 * d * case["rank"]
        return {"bytes": 4.0 * params + 8.0 * m.num_layers * 2.0 * d * case["rank"] + 16.0 * tokens, "flops": 2.0 * dense + 3.0 * low + 3.5 * attn}
    out = {"score": 4.0 * tokens, "sliding": 0.0, "logits": 4.0 * tokens * m.vocab_size}[kind]
    return {"bytes": 4.0 * params + 16.0 * tokens + out, "flops": dense + attn}


def tolerance(case):
    """Measured against the autograd model in fp32 (weights after the step, gradients, losses) and, for GPTQ, against the fp32 row
    algorithm with its trailing sums in another order; about four times the largest value seen."""
    kind = case["kind"]
    if kind == "gptq":
        return {"rel": 1e-3, "differ": 0.002}
    if kind == "sliding":
        return {"rel": 3e-4}
    if kind == "score":
        return {"rel": 0.006, "max": 0.04}
    if kind == "logits":
        return {"rel": 0.03, "max": 0.25}
    if kind == "train":
        return {"rel": 1e-3, "max": 0.02}
    return {"rel": 0.03, "max": 0.9}
