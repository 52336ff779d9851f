"""What users have this framework do on one GPU, as measurable cases.

A case is a dict of plain values.  `prepare` builds what a program holds before the call (model, optimizer, batches on
the GPU), `run` makes one pass through the public entry points and returns everything that pass computes, `work` gives
the bytes and operations the pass cannot do without, and `tolerance` how far another correct implementation may differ.

Kinds of cases
  train          Engine.train_step: gradient accumulation over micro-batches, clipping, AdamW
  score          a labelled packed batch through the engine's model without gradients: loss and hidden states
  logits         one prompt through a plain model without gradients: hidden states and logits
  moe            the dropless MoE layer on its own (it is a drop-in for other models): forward and backward
  attention      causal grouped-query attention over packed sequences: forward and backward
  expert_linear  parallel_linear_lora, the grouped linear with per-expert adapters: forward and backward

Weights are those of a model that has been trained for a while rather than of a fresh one where that matters: tokens
are routed with a clear preference (embeddings carry a component along the router rows of their two experts, experts
differ in popularity), matrices that write to the residual stream are scaled down with depth, and adapters are the ones
of a resumed run (neither factor is zero).
"""
import math
import random

import torch

from moe_distributed_training_b200 import MixtralConfig, ops
from moe_distributed_training_b200.config import LoraConfig, MoEArguments
from moe_distributed_training_b200.data.synthetic import collate_packed
from moe_distributed_training_b200.models.mixtral import MixtralForCausalLM
from moe_distributed_training_b200.moe.layer import dMoE
from moe_distributed_training_b200.optim.adamw import FusedAdamW
from moe_distributed_training_b200.optim.schedulers import get_scheduler
from moe_distributed_training_b200.parallel.fsdp import ShardedMixtral
from moe_distributed_training_b200.peft.lora import get_peft_model
from moe_distributed_training_b200.train.engine import Engine, lora_targets
from scattermoe_utils.parallel_linear_lora import parallel_linear_lora

DEV, BF16 = "cuda", torch.bfloat16
LORA_R, LORA_ALPHA = 16, 32
IGNORE = -100

# widths: "8x7b" is MixtralConfig's default, "small" the toy model of the smoke test
WIDTHS = {"8x7b": dict(vocab=32000, hidden=4096, ffn=14336, heads=32, kv=8, experts=8, topk=2),
          "small": dict(vocab=2048, hidden=512, ffn=1024, heads=4, kv=2, experts=4, topk=2)}


def listed():
    return [
        # --- training steps
        # trying a configuration out on a toy model: many short kernels, so launches and host work decide
        {"name": "train-toy", "kind": "train", "width": "small", "layers": 2, "lora": "none", "micro": 2, "seqs": 1,
         "lo": 128, "hi": 256, "recompute": True},
        # the benchmark's step (LoRA on attention, one sequence of 128-1024 tokens per micro-batch) on the two-layer
        # model that the entry script's truncation flag gives
        {"name": "train-lora-attn", "kind": "train", "width": "8x7b", "layers": 2, "lora": "attn-only", "micro": 4, "seqs": 1,
         "lo": 128, "hi": 1024, "recompute": True},
        # the same with per-expert adapters
        {"name": "train-lora-all", "kind": "train", "width": "8x7b", "layers": 2, "lora": "all", "micro": 4, "seqs": 1,
         "lo": 128, "hi": 1024, "recompute": True},
        # full fine-tuning: weight gradients of every matrix, and the optimizer over all of them (one layer, since what
        # comes back is every weight and both moments)
        {"name": "train-full", "kind": "train", "width": "8x7b", "layers": 1, "lora": "none", "micro": 4, "seqs": 1,
         "lo": 128, "hi": 1024, "recompute": True},
        # a large per-device batch of longer sequences, activations kept: compute bound
        {"name": "train-lora-packed", "kind": "train", "width": "8x7b", "layers": 1, "lora": "attn-only", "micro": 1, "seqs": 6,
         "lo": 512, "hi": 2048, "recompute": False},
        # --- inference-like passes
        # evaluation loss over a packed batch of ragged sequences
        {"name": "score-packed", "kind": "score", "width": "8x7b", "layers": 2, "seqs": 16, "lo": 128, "hi": 1024},
        # one short prompt: every expert's weights are read for a handful of rows
        {"name": "logits-prompt", "kind": "logits", "width": "8x7b", "layers": 2, "tokens": 77},
        # --- single operators
        # the MoE layer inside another model, trainable experts, large batch
        {"name": "moe-large", "kind": "moe", "width": "8x7b", "tokens": 12000, "train": True},
        # attention of one instruction example, and of long documents
        {"name": "attention-short", "kind": "attention", "heads": 32, "kv": 8, "seqs": 1, "lo": 613, "hi": 613},
        {"name": "attention-long", "kind": "attention", "heads": 32, "kv": 8, "seqs": 4, "lo": 1024, "hi": 8192},
        # the grouped linear with adapters, up and (gate-weighted) down
        {"name": "expert-linear-up", "kind": "expert_linear", "tokens": 576, "experts": 8, "topk": 2, "k": 4096, "n": 14336, "gates": False},
        {"name": "expert-linear-down", "kind": "expert_linear", "tokens": 3001, "experts": 4, "topk": 2, "k": 14336, "n": 4096, "gates": True},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["train", "train", "train", "score", "logits", "moe", "attention", "attention", "expert_linear"])
    if kind == "train":
        if rng.random() < 0.25:
            lo = _log_int(rng, 16, 256)
            return {"kind": "train", "width": "small", "layers": rng.randint(1, 3), "lora": rng.choice(["none", "attn-only", "all"]),
                    "micro": rng.randint(1, 4), "seqs": rng.randint(1, 3), "lo": lo, "hi": 2 * lo, "recompute": rng.random() < 0.7}
        lo = _log_int(rng, 64, 512)
        return {"kind": "train", "width": "8x7b", "layers": 1, "lora": rng.choice(["none", "attn-only", "all"]),
                "micro": rng.randint(1, 4), "seqs": rng.randint(1, 2), "lo": lo, "hi": 2 * lo, "recompute": rng.random() < 0.7}
    if kind == "score":
        return {"kind": "score", "width": "8x7b", "layers": rng.randint(1, 2), "seqs": rng.randint(1, 16), "lo": _log_int(rng, 32, 256), "hi": 1024}
    if kind == "logits":
        return {"kind": "logits", "width": "8x7b", "layers": rng.randint(1, 2), "tokens": _log_int(rng, 1, 1024)}
    if kind == "moe":
        return {"kind": "moe", "width": rng.choice(["8x7b", "8x7b", "small"]), "tokens": _log_int(rng, 16, 12000), "train": rng.random() < 0.6}
    if kind == "attention":
        kv = rng.choice([2, 4, 8])
        lo = _log_int(rng, 64, 2048)
        return {"kind": "attention", "heads": kv * rng.choice([1, 2, 4]), "kv": kv, "seqs": rng.randint(1, 5), "lo": lo, "hi": 2 * lo}
    k, n = rng.choice([(4096, 14336), (14336, 4096), (1024, 3584), (512, 1024)])
    return {"kind": "expert_linear", "tokens": _log_int(rng, 16, 4096), "experts": rng.choice([1, 2, 4, 8]), "topk": 2 if rng.random() < 0.8 else 1,
            "k": k, "n": n, "gates": rng.random() < 0.5}


# ---------------------------------------------------------------------------------------------------------------------
# sizes that follow from a case (the same for every seed)
# ---------------------------------------------------------------------------------------------------------------------
def _lengths(case):
    """Sequence lengths of every micro-batch, uniform in [lo, hi] as instruction examples are."""
    rng = random.Random("%s" % sorted((k, v) for k, v in case.items() if k != "name"))
    return [[rng.randint(case["lo"], case["hi"]) for _ in range(case["seqs"])] for _ in range(case.get("micro", 1))]


# ---------------------------------------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------------------------------------
class _Rand:
    def __init__(self, seed):
        self.gen = torch.Generator(device=DEV).manual_seed(int(seed) % (1 << 62))

    def normal(self, *shape, std=1.0):
        return torch.empty(*shape, dtype=BF16, device=DEV).normal_(0.0, std, generator=self.gen)

    def fill(self, t, std):
        with torch.no_grad():
            t.normal_(0.0, std, generator=self.gen)

    def ints(self, high, *shape):
        return torch.randint(0, high, shape, device=DEV, generator=self.gen)

    def uniform(self, *shape):
        return torch.rand(*shape, device=DEV, generator=self.gen)


@torch.no_grad()
def _routed(r, x, router_w, topk):
    """x plus, for every row, a component along the router rows of `topk` experts of its own, popular ones more often."""
    experts = router_w.shape[0]
    popularity = torch.softmax(0.5 * torch.randn(experts, device=DEV, generator=r.gen), 0)
    chosen = torch.multinomial(popularity.expand(x.shape[0], experts), topk, generator=r.gen)
    direction = torch.nn.functional.normalize(router_w.float(), dim=1)
    for c in range(topk):
        x = x + (9.0 + 2.0 * r.uniform(x.shape[0], 1)) * direction[chosen[:, c]]
    return x


def _config(case):
    w = WIDTHS[case["width"]]
    return MixtralConfig(vocab_size=w["vocab"], hidden_size=w["hidden"], intermediate_size=w["ffn"], num_hidden_layers=case["layers"],
                         num_attention_heads=w["heads"], num_key_value_heads=w["kv"], head_dim=128, num_local_experts=w["experts"],
                         num_experts_per_tok=w["topk"])


def _model(case, r):
    cfg = _config(case)
    model = MixtralForCausalLM(cfg, dtype=BF16, device="meta").to_empty(device=DEV)
    out_std = 0.02 / math.sqrt(2.0 * max(cfg.num_hidden_layers, 2))
    with torch.no_grad():
        for name, p in model.named_parameters():
            if "norm" in name:
                p.fill_(1.0)
            else:
                r.fill(p, out_std if name.endswith(("o_proj.weight", "w2")) else 0.02)
        table = r.normal(cfg.vocab_size, cfg.hidden_size).float()
        for layer in model.model.layers:
            table = _routed(r, table, layer.block_sparse_moe.router.layer.weight, cfg.num_experts_per_tok)
        model.model.embed_tokens.weight.copy_(table)
    return cfg, model


def _engine(case, r):
    """What `build_engine` puts together, on weights of our own."""
    cfg, model = _model(case, r)
    targets = lora_targets(case.get("lora", "none"), True)
    if targets is not None:
        get_peft_model(model, LoraConfig(r=LORA_R, lora_alpha=LORA_ALPHA, target_modules=targets), adapter_dtype=BF16)
        for name, p in model.named_parameters():
            if "lora_B" in name:
                r.fill(p, 0.01)
            elif "lora_A" in name:
                r.fill(p, 0.01)
    runner = ShardedMixtral(model, recompute=case.get("recompute", True))
    params = [p for p in model.parameters() if p.requires_grad]
    opt = FusedAdamW(params, lr=5e-5, weight_decay=0.01)
    sched = get_scheduler("linear", opt, 0, 10_000_000)
    return cfg, Engine(model, runner, opt, sched, None, torch.device(DEV, torch.cuda.current_device()), 0, 1, 1, max_grad_norm=1.0)


def _batch(cfg, lens, r):
    """One packed micro-batch; the first 40 % of every sequence is prompt and carries no label."""
    examples = []
    for n in lens:
        ids = r.ints(cfg.vocab_size, n)
        labels = ids.clone()
        labels[: int(0.4 * n)] = IGNORE
        examples.append({"input_ids": ids, "labels": labels})
    mb = collate_packed(examples)
    mb["cu_seqlens"] = mb["cu_seqlens"].to(DEV)
    return mb


def prepare(case, seed):
    r, kind = _Rand(seed), case["kind"]
    if kind == "train":
        cfg, engine = _engine(case, r)
        return {"kind": kind, "engine": engine, "batches": [_batch(cfg, lens, r) for lens in _lengths(case)]}
    if kind == "score":
        cfg, engine = _engine(case, r)
        return {"kind": kind, "engine": engine, "batch": _batch(cfg, _lengths(case)[0], r)}
    if kind == "logits":
        cfg, model = _model(case, r)
        return {"kind": kind, "model": model, "ids": r.ints(cfg.vocab_size, 1, case["tokens"])}
    if kind == "moe":
        w = WIDTHS[case["width"]]
        layer = dMoE(MoEArguments(hidden_size=w["hidden"], ffn_hidden_size=w["ffn"], moe_num_experts=w["experts"], moe_top_k=w["topk"],
                                  bf16=True, device=DEV))
        for name, p in layer.named_parameters():
            r.fill(p, 0.02)
            p.requires_grad_(case["train"])
        x = _routed(r, r.normal(case["tokens"], w["hidden"]).float(), layer.router.layer.weight, w["topk"])
        x = (x / x.square().mean(1, keepdim=True).sqrt()).to(BF16)[None]
        return {"kind": kind, "layer": layer, "x": x.requires_grad_(True), "dy": r.normal(1, case["tokens"], w["hidden"], std=0.1)}
    if kind == "attention":
        lens = _lengths(case)[0]
        T, d = sum(lens), 128
        cu = torch.tensor([sum(lens[:i]) for i in range(len(lens) + 1)], dtype=torch.int32, device=DEV)
        q, k, v = (r.normal(T, h, d).requires_grad_(True) for h in (case["heads"], case["kv"], case["kv"]))
        return {"kind": kind, "qkv": (q, k, v), "cu": cu, "max": max(lens), "do": r.normal(T, case["heads"], d)}
    T, k, E = case["tokens"], case["topk"], case["experts"]
    popularity = torch.softmax(0.5 * torch.randn(E, device=DEV, generator=r.gen), 0)
    chosen = torch.multinomial(popularity.expand(T, E), min(k, E), generator=r.gen)
    chosen = chosen.repeat(1, k)[:, :k]          # (one expert: both choices are it)
    sorted_ids, order = torch.sort(chosen.reshape(-1), stable=True)
    x = r.normal(T, case["k"]).requires_grad_(True)
    W = r.normal(E, case["k"], case["n"], std=0.02)
    A, B = (r.normal(E, *s, std=0.01).requires_grad_(True) for s in ((case["k"], LORA_R), (LORA_R, case["n"])))
    gates = None
    if case["gates"]:
        gates = torch.softmax(r.normal(T, k).float(), 1).to(BF16).requires_grad_(True)
    rows = T if case["gates"] else T * k
    return {"kind": kind, "x": x, "W": W, "A": A, "B": B, "gates": gates, "topk": k, "ids": sorted_ids, "order": order,
            "dy": r.normal(rows, case["n"], std=0.1)}


# ---------------------------------------------------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------------------------------------------------
def run(s):
    kind = s["kind"]
    if kind == "train":
        engine = s["engine"]
        stats = engine.train_step(s["batches"])
        trained = [p for p in engine.model.parameters() if p.requires_grad]
        state = [engine.optimizer.state[p] for p in trained]
        return {"loss": stats["loss"], "grad_norm": stats["grad_norm"], "params": [p.detach() for p in trained],
                "exp_avg": [st["exp_avg"] for st in state], "exp_avg_sq": [st["exp_avg_sq"] for st in state]}
    if kind == "score":
        b = s["batch"]
        with torch.no_grad():
            out = s["engine"].model(b["input_ids"], labels=b["labels"], cu_seqlens=b["cu_seqlens"], max_seqlen=b["max_seqlen"])
        return {"loss": out.loss, "hidden": out.hidden_states, "tokens": out.num_tokens}
    if kind == "logits":
        with torch.no_grad():
            out = s["model"](s["ids"], return_logits=True)
        return {"hidden": out.hidden_states, "logits": out.logits}
    if kind == "moe":
        layer, x = s["layer"], s["x"]
        layer.zero_grad(set_to_none=True)
        x.grad = None
        y, _ = layer(x)
        y.backward(s["dy"])
        grads = {n: p.grad for n, p in layer.named_parameters() if p.grad is not None}
        return {"y": y.detach(), "dx": x.grad, "grads": grads}
    if kind == "attention":
        o = ops.attention(*s["qkv"], s["cu"], s["max"])
        return {"o": o.detach(), "grads": list(torch.autograd.grad(o, s["qkv"], s["do"]))}
    y = parallel_linear_lora(s["x"], s["W"], s["A"], s["B"], LORA_R, LORA_ALPHA, s["topk"], s["ids"], s["order"], gates=s["gates"])
    wrt = [s["x"], s["A"], s["B"]] + ([s["gates"]] if s["gates"] is not None else [])
    return {"y": y.detach(), "grads": list(torch.autograd.grad(y, wrt, s["dy"]))}


# ---------------------------------------------------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------------------------------------------------
def _attention_flops(lens, heads, d=128):
    return sum(2.0 * n * n for n in lens) * d * heads          # the causal half of Q K^T and of P V


def work(case):
    kind = case["kind"]
    if kind in ("train", "score", "logits"):
        w, L = WIDTHS[case["width"]], case["layers"]
        H, F, V, E, k = w["hidden"], w["ffn"], w["vocab"], w["experts"], w["topk"]
        batches = [[case["tokens"]]] if kind == "logits" else _lengths(case)
        attn = 2 * H * 128 * (w["heads"] + w["kv"])
        layer = attn + E * H + 3 * E * H * F
        full, lora = case.get("lora") == "none", case.get("lora") in ("attn-only", "all")
        adapters = 0
        if lora:
            adapters += LORA_R * (2 * (H + 128 * w["heads"]) + 2 * (H + 128 * w["kv"]))
            if case["lora"] == "all":
                adapters += 3 * E * LORA_R * (H + F)
        flops = nbytes = 0.0
        for lens in batches:
            T = sum(lens)
            used = min(1.0, T * k / E) if T * k < E else 1.0          # a single token reads the weights of k experts
            scored = T if kind == "logits" else sum(n - int(0.4 * n) for n in lens)
            fwd = L * (2.0 * T * (attn + E * H + 3 * H * F * k) + _attention_flops(lens, w["heads"])) + 2.0 * scored * H * V
            read = 2.0 * (L * (attn + E * H + 3 * E * H * F * used) + H * V + T * H)
            write = 2.0 * T * H + (2.0 * T * V if kind == "logits" else 0)
            if kind == "train":
                # gradients by the inputs cost what the forward costs (attention 2.5 times that); by the weights again
                bwd = L * (2.0 * T * (attn + E * H + 3 * H * F * k) + 2.5 * _attention_flops(lens, w["heads"])) + 2.0 * scored * H * V
                if full:
                    bwd += L * 2.0 * T * (attn + E * H + 3 * H * F * k) + 2.0 * scored * H * V
                fwd, read = fwd + bwd, 2 * read
            flops, nbytes = flops + fwd, nbytes + read + write
        if kind == "train":
            trained = (L * layer + 2 * V * H) if full else L * adapters
            nbytes += 2.0 * trained * 8          # the gradient is written and read, weight and moments are read and written
        return {"bytes": nbytes, "flops": flops}
    if kind == "moe":
        w, T = WIDTHS[case["width"]], case["tokens"]
        P = 3 * w["experts"] * w["hidden"] * w["ffn"]
        one = 2.0 * T * w["topk"] * 3 * w["hidden"] * w["ffn"]
        return {"flops": one * (3 if case["train"] else 2), "bytes": 2.0 * (P * (3 if case["train"] else 2) + 4 * T * w["hidden"])}
    if kind == "attention":
        lens = _lengths(case)[0]
        return {"flops": 3.5 * _attention_flops(lens, case["heads"]), "bytes": 2.0 * sum(lens) * 128 * (4 * case["heads"] + 4 * case["kv"])}
    M, K, N, E, r = case["tokens"] * case["topk"], case["k"], case["n"], case["experts"], LORA_R
    out = case["tokens"] if case["gates"] else M
    return {"flops": 2.0 * M * K * N * 2 + 2.0 * M * r * (K + N) * 3,
            "bytes": 2.0 * (2 * E * K * N + 2 * case["tokens"] * K + 2 * out * N + 4 * E * r * (K + N))}


def tolerance(case):
    # bf16 inputs, intermediates and results (each rounding up to 0.4 %), sums in fp32.  About four times the distance to
    # the same path on torch's library operators (`ops.set_backend("library")`); a training step's second moments are the
    # furthest off (0.022), the gradient having passed two layers twice.  "max" of the steps: single elements of a
    # gradient that nearly cancels.
    if case["kind"] == "train":
        return {"rel": 0.03, "max": 0.95}
    if case["kind"] in ("score", "logits", "moe"):
        return {"rel": 0.03, "max": 0.5}                 # seen 0.011 / 0.14 (score), 0.010 / 0.08 (logits), 0.013 / 0.13 (moe)
    if case["kind"] == "attention":
        return {"rel": 0.015, "max": 0.4}                # seen 0.0037 / 0.12
    return {"rel": 0.015, "max": 0.15}                   # seen 0.0038 / 0.033
