"""The workloads whose speed this framework is judged by, on one GPU, through its public entry points.

  listed()   the named cases;  draw(rng)  one more case of the same ranges
  prepare()  what a training program holds before it calls: model, wrapper, optimizer, recorded step, batch
  run()      one pass (one step, one evaluation, one operator forward + backward, one optimizer update)
  work()     bytes and floating-point operations that a pass cannot do without
  tolerance()  how far two correct implementations at the same precision may be apart

Five kinds of pass:
  train       a whole training step (forward, backward, gradient reduction, AdamW) under DDP, ZeRO-2 or ZeRO-3 in a group
              of one, recorded as a CUDA graph or issued eagerly.  A group of one is one rank's share of a larger job.
  eval        logits and loss without gradients
  attention   the causal-attention operator, forward and backward
  projection  the linear operator, forward and backward
  optimizer   one AdamW update of a flat parameter shard
Token ids are uniform in [0, vocab) and weights are the model's own initialisation: the data the benchmark uses.
"""

import math
import weakref

import torch

import tandem_b200
from tandem_b200 import ops
from tandem_b200.ddp import DDP, BucketAdamW
from tandem_b200.model import GPT, Config
from tandem_b200.models.gpt import loss_fn
from tandem_b200.optim import ShardedAdamW
from tandem_b200.parallel.graph import GraphedStep
from tandem_b200.zero import FSDP, ZeRO

# The learning rate of the first step of a linear warm-up to 3e-4 over 100 steps: the weights stay at their
# initialisation, so that a pass can be repeated and two implementations stay comparable after several steps.
LR, WEIGHT_DECAY = 3e-6, 0.1


def _train(name, layers, dim, heads, vocab, seq, batch, strategy, graph):
    return {"name": name, "kind": "train", "layers": layers, "dim": dim, "heads": heads, "vocab": vocab, "seq": seq, "batch": batch,
            "strategy": strategy, "graph": graph}


def listed():
    return [
        # A model of two small blocks, every kernel issued from Python: first contact, unit-sized experiments.
        _train("train_2layer_eager", 2, 256, 4, 65, 128, 4, "ddp", False),
        # The 11M-parameter preset under ZeRO-2, a laptop-sized job: every kernel is a few microseconds.
        _train("train_small_zero2", 6, 384, 6, 256, 256, 12, "zero2", True),
        # The 85.8M-parameter flagship, one rank's share of a global batch of 16 x 512 tokens on 8 GPUs.
        _train("train_medium_1024", 12, 768, 12, 65, 512, 2, "ddp", True),
        # The flagship benchmark itself: 16 x 512 tokens on one GPU.
        _train("train_medium_8192", 12, 768, 12, 65, 512, 16, "ddp", True),
        # The 24-layer pipeline configuration with its 50k vocabulary, one micro-batch of 4 x 1024 tokens.
        _train("train_24layer_4096", 24, 1024, 16, 50304, 1024, 4, "ddp", True),
        # The 1.3B-parameter model under ZeRO-3, one rank's share of a global batch of 64 x 2048 tokens on 8 GPUs.
        _train("train_1p3b_16384", 24, 2048, 16, 50304, 2048, 8, "zero3", False),
        # Validation loss of the 302M-parameter preset over a last, short batch.
        {"name": "eval_large_5x512", "kind": "eval", "layers": 24, "dim": 1024, "heads": 16, "vocab": 256, "seq": 512, "batch": 5},
        # Attention over sequences longer than the presets', where it outweighs the projections.
        {"name": "attention_4096", "kind": "attention", "batch": 2, "seq": 4096, "heads": 16, "head_dim": 128},
        # A projection whose rows and output width fit no tile.
        {"name": "projection_ragged", "kind": "projection", "rows": 1537, "inner": 768, "outer": 1003, "bias": True},
        # The AdamW update of one rank's fp32 shard, of an odd length as torch.tensor_split leaves it.
        {"name": "optimizer_fp32_shard", "kind": "optimizer", "elements": 42921217, "dtype": "float32"},
    ]


def _log_int(rng, lo, hi, step=1):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / step)) * step))


def draw(rng):
    most = work(listed()[5])["flops"]
    kind = rng.choices(["train", "eval", "attention", "projection", "optimizer"], [5, 2, 2, 2, 1])[0]
    if kind == "attention":
        head_dim = rng.choice([64, 128])
        seq = _log_int(rng, 128, 8192, 128)
        heads = rng.randint(2, 16)
        return {"kind": kind, "batch": _log_int(rng, 1, max(1, min(64, 32768 // seq))), "seq": seq, "heads": heads, "head_dim": head_dim}
    if kind == "projection":
        return {"kind": kind, "rows": _log_int(rng, 16, 16384), "inner": _log_int(rng, 64, 8192, 8), "outer": _log_int(rng, 60, 8192),
                "bias": rng.random() < 0.5}
    if kind == "optimizer":
        return {"kind": kind, "elements": _log_int(rng, 1 << 14, 1 << 26), "dtype": rng.choice(["float32", "bfloat16"])}
    while True:
        head_dim = rng.choice([64, 64, 128])
        heads = rng.randint(2, 2048 // head_dim)
        seq = _log_int(rng, 128, 2048, 128)
        case = {"kind": kind, "layers": _log_int(rng, 2, 24), "dim": heads * head_dim, "heads": heads, "vocab": _log_int(rng, 61, 50304),
                "seq": seq, "batch": _log_int(rng, 1, max(1, 16384 // seq))}
        if kind == "train":
            case["strategy"] = rng.choice(["ddp", "ddp", "zero2", "zero3"])
            # a recorded step keeps its activations: large ones are issued eagerly
            case["graph"] = rng.random() < 0.75 and 32 * case["layers"] * case["dim"] * seq * case["batch"] < 8e9
        if work(case)["flops"] <= most:
            return case


# ------------------------------------------------------------------------------------------ what a program holds
class Training:
    """One training job in a group of one."""

    def __init__(self, case, seed):
        self.group = tandem_b200.Group.from_env(device="cuda")
        model = _model(case, seed)
        x, y = self.batch = _tokens(case, seed)
        graph, strategy = case["graph"], case["strategy"]
        if strategy == "ddp":
            self.wrapper = DDP(model, self.group, rebuild=False)
            self.optimizer = BucketAdamW(self.wrapper, lr=LR, weight_decay=WEIGHT_DECAY, during_backward=True)
        else:
            adam = ShardedAdamW(lr=LR, weight_decay=WEIGHT_DECAY)
            if strategy == "zero2":
                self.wrapper = ZeRO(model, self.group, 2, adam, capturable=graph)
            else:
                self.wrapper = FSDP(model, self.group, adam, capturable=graph)
            self.optimizer = self.wrapper
        _open.append((weakref.ref(self), self.group, [self.wrapper, self.optimizer, model]))
        self.recorded = GraphedStep(self.wrapper, self.optimizer, x, y) if graph else None

    def step(self):
        x, y = self.batch
        if self.recorded is not None:
            return self.recorded(x, y)
        self.optimizer.zero_grad()
        loss = self.wrapper(x, y)
        loss.backward()
        self.optimizer.step()
        return loss.detach()

    def results(self):
        """The tensors that hold the step's gradients (or the moments they went into), unit by unit, and the updated weights."""
        w = self.wrapper
        if isinstance(w, DDP):
            (arena,) = w.arenas.values()
            first = self.optimizer.slots[0]["flat"]  # a slice of the one buffer that holds all weights
            weights = first.as_strided((arena.flat.numel(),), (1,), 0)
            return _by_unit(w.module, arena.flat, arena.where), [weights]
        if isinstance(w, ZeRO):
            _, mean, square = w.opt.state["flat"]
            return _by_unit(w.module, mean, w.flat.offset), [square, w.buf]
        if self.recorded is not None:
            return [w.opt.state[u.index][1] for u in w.units], [u.shard for u in w.units]
        return [u.grad_shard for u in w.units], [u.shard for u in w.units]


def _by_unit(model, flat, offset):
    """The slices of a flat buffer that belong to the model's units (each contiguous in it)."""
    out = []
    for unit in model.units():
        ends = [(offset[p], offset[p] + p.numel()) for p in unit.parameters()]
        out.append(flat[min(a for a, _ in ends):max(b for _, b in ends)])
    return out


_open = []  # (job, its group, what its parameters' hooks keep alive)


def _close_finished():
    """Ends the jobs nobody holds any more: closes their groups and drops what the gradient hooks would keep alive."""
    for entry in [e for e in _open if e[0]() is None]:
        _open.remove(entry)
        _, group, held = entry
        group.close()
        for thing in held:
            thing.__dict__.clear()
    if torch.cuda.memory_reserved() > 64 << 30:
        torch.cuda.empty_cache()


def _model(case, seed):
    torch.manual_seed(seed)
    with torch.device("cuda"):
        model = GPT(Config(vocab=case["vocab"], seq=case["seq"], layers=case["layers"], heads=case["heads"], dim=case["dim"],
                           kernels="b200"))
    return model.bfloat16()


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _tokens(case, seed):
    rows = torch.randint(0, case["vocab"], (case["batch"], case["seq"] + 1), generator=_generator(seed), device="cuda")
    return rows[:, :-1].contiguous(), rows[:, 1:].contiguous()


def _normal(gen, *shape, std=1.0, dtype=torch.bfloat16):
    return (torch.randn(*shape, generator=gen, device="cuda") * std).to(dtype)


def prepare(case, seed):
    _close_finished()
    kind = case["kind"]
    if kind == "train":
        return {"kind": kind, "job": Training(case, seed)}
    gen = _generator(seed)
    if kind == "eval":
        return {"kind": kind, "model": _model(case, seed), "batch": _tokens(case, seed)}
    if kind == "attention":
        B, T, d = case["batch"], case["seq"], case["heads"] * case["head_dim"]
        # LayerNorm output (unit variance) through N(0, 0.02) weights gives q, k and v of this spread early in training
        return {"kind": kind, "heads": case["heads"], "qkv": _normal(gen, B, T, 3 * d, std=0.02 * math.sqrt(d)).requires_grad_(),
                "grad": _normal(gen, B, T, d, std=1e-3)}
    if kind == "projection":
        M, K, N = case["rows"], case["inner"], case["outer"]
        return {"kind": kind, "x": _normal(gen, M, K).requires_grad_(), "w": _normal(gen, N, K, std=0.02).requires_grad_(),
                "b": _normal(gen, N, std=0.02).requires_grad_() if case["bias"] else None, "grad": _normal(gen, M, N, std=1e-3)}
    n, dtype = case["elements"], getattr(torch, case["dtype"])
    rule, shard = ShardedAdamW(lr=LR, weight_decay=WEIGHT_DECAY), _normal(gen, n, std=0.02, dtype=dtype)
    rule.ensure_state("flat", shard)
    return {"kind": kind, "rule": rule, "shard": shard, "grad": _normal(gen, n, std=1e-3, dtype=dtype)}


def run(state):
    kind = state["kind"]
    if kind == "train":
        loss = state["job"].step()
        gradients, weights = state["job"].results()
        return [loss, *gradients, *weights]
    if kind == "eval":
        x, y = state["batch"]
        with torch.no_grad():
            logits = state["model"](x)
            return [logits, loss_fn(logits, y, "b200")]
    if kind == "attention":
        qkv = state["qkv"]
        out = ops.causal_attention(qkv, state["heads"])
        return [out.detach(), *torch.autograd.grad(out, [qkv], state["grad"])]
    if kind == "projection":
        x, w, b = state["x"], state["w"], state["b"]
        y = ops.linear(x, w, b)
        return [y.detach(), *torch.autograd.grad(y, [x, w] if b is None else [x, w, b], state["grad"])]
    rule, shard = state["rule"], state["shard"]
    rule.update("flat", shard, state["grad"])
    return [shard, *rule.state["flat"][1:]]


# ------------------------------------------------------------------------------------------ what a pass cannot do without
def work(case):
    kind = case["kind"]
    if kind == "optimizer":
        n = case["elements"]
        # gradient in, both moments and the fp32 weights in and out, and with 16-bit weights their rounded copy out
        return {"bytes": n * (4 + 24) if case["dtype"] == "float32" else n * (2 + 24 + 2), "flops": 15 * n}
    if kind == "projection":
        M, K, N = case["rows"], case["inner"], case["outer"]
        return {"bytes": 2 * (2 * M * K + 2 * N * K + 2 * M * N + (2 * N if case["bias"] else 0)), "flops": 6 * M * K * N}
    if kind == "attention":
        B, T, H, D = case["batch"], case["seq"], case["heads"], case["head_dim"]
        # causal half of two products forward and five backward; qkv, out, d_out and d_qkv once each
        return {"bytes": 2 * B * T * H * D * 8, "flops": 7 * B * H * T * T * D}
    L, d, V, B, T = (case[k] for k in ("layers", "dim", "vocab", "batch", "seq"))
    matrices = L * 12 * d * d + V * d
    params = matrices + L * 13 * d + V * d + T * d + 2 * d
    forward = 2 * B * T * matrices + L * 2 * B * T * T * d
    if kind == "eval":
        return {"bytes": 2 * params + 2 * B * T * V + 16 * B * T, "flops": forward}
    # bf16 weights in and out, bf16 gradients out, fp32 master weights and both moments in and out
    return {"bytes": 30 * params + 16 * B * T, "flops": 2 * B * T * matrices * 3 + L * 7 * B * T * T * d}


def tolerance(case):
    """Measured against the same model on torch's bf16 operators (cuBLAS, SDPA): gradients differ by up to 1.5e-2 in norm and
    logits by 1.4e-2; single gradients differ by up to about the root mean square of their unit, because a few rows of a large
    embedding and the biases of a block have gradients far above it.  Attention against exact scores: 2.3e-3 and 0.11; the
    projection against cuBLAS: 3e-3 and 0.016."""
    kind = case["kind"]
    if kind == "optimizer":
        return {"rel": 1e-5} if case["dtype"] == "float32" else {"rel": 1e-4, "max": 1e-2}
    if kind == "attention":
        return {"rel": 1e-2, "max": 0.4}
    if kind == "projection":
        return {"rel": 1e-2, "max": 0.06}
    return {"rel": 2e-2, "max": 0.95}
