"""The training steps this framework is timed on, on one B200.

What a user of the framework does with it, over and over, is `QwenTrainer.train_step`: tokens in,
micro-batches through the sharded runtime (parameter gathers, forward, backward, gradient
reductions), the optimizer update, the loss read back.  Every case is one such step through the
public API (`Qwen2CausalLM` -> `ShardedRuntime.register` -> `QwenTrainer`), so each covers forward,
backward and update; they differ in model widths, depth, batch, sequence length, accumulation,
padding, optimizer, dtype and runtime switches.

Sizes are those of `configs/*.yaml`, `bench.py` and the tests.  Where a model is too large for
three copies of its training state on one GPU, a case takes a *slice* of it: fewer layers and the
vocabulary cut in the same proportion, so that the LM head keeps the share of the step it has in
the whole model.
"""

import gc
import math

import torch

from shardtrain_b200.models.qwen2 import Qwen2CausalLM, Qwen2ModelConfig
from shardtrain_b200.runtime.engine import ShardedRuntime
from shardtrain_b200.training.qwen2_trainer import QwenTrainer

BASE = dict(
    heads=2, kv_heads=1, head_dim=128, inter=512, layers=2, vocab=2048, tied=True,
    batch=4, seq=256, accum=2,
    dtype="bf16", optimizer="adamw",
    padding="none",        # none | ones (an all-ones key mask) | right | left (ragged samples)
    positions="default",   # default | row ([1, S] given) | sample ([B, S] given)
    overlap=True,          # prefetch / asynchronous reduction switches, as the B200 configs set them
    diagnostics=False,     # the runtime's event log
)


def _case(name, **fields):
    return {"name": name, **BASE, **fields}


WIDTH_1P5B = dict(heads=12, kv_heads=2, inter=8960)       # configs/qwen25_1p5b_config.yaml
WIDTH_7B = dict(heads=28, kv_heads=4, inter=18944)        # configs/qwen25_7b_config.yaml


def listed():
    return [
        # the two-layer model of the smoke entry point and the GPU tests: launch and host latency
        _case("smoke"),
        # shortest useful call: one short sequence, no accumulation, plain SGD, untied head (the
        # shapes of the end-to-end tests with the runtime's default switches and event log)
        _case("short_sgd", batch=1, seq=128, accum=1, optimizer="sgd", tied=False, overlap=False,
              diagnostics=True),
        # what each GPU of the 8-GPU headline run computes per step: one sequence per micro-step
        # (a quarter of the 1.5B model)
        _case("rank_of_8_1p5b", **WIDTH_1P5B, layers=7, vocab=37984, batch=2, seq=512,
              padding="ones", positions="row"),
        # the headline benchmark itself: Qwen2.5-1.5B, all 28 layers, S512, global batch 16, 2
        # micro-steps, inputs as bench.py passes them
        _case("headline_1p5b", **WIDTH_1P5B, layers=28, vocab=151936, batch=16, seq=512,
              padding="ones", positions="row"),
        # ragged fine-tuning batch at 1.5B widths: odd length, right-padded samples, ignored labels
        _case("padded_1p5b", **WIDTH_1P5B, layers=7, vocab=37984, batch=6, seq=777, accum=3,
              padding="right", positions="sample"),
        # long documents at 1.5B widths: attention is the larger part of the layer
        _case("long_1p5b", **WIDTH_1P5B, layers=7, vocab=37984, batch=2, seq=8192),
        # full vocabulary over few layers: the LM head and its loss are the larger part
        _case("head_1p5b", **WIDTH_1P5B, layers=2, vocab=151936, batch=8, seq=512,
              padding="ones", positions="row"),
        # 7B widths at the 7B config's micro-batch (4 x 2048), untied head (a seventh of the model)
        _case("slice_7b", **WIDTH_7B, layers=4, vocab=21728, tied=False, batch=8, seq=2048,
              padding="ones", positions="row"),
        # a small pre-training model, left-padded, SGD, no accumulation, plain switches
        _case("mid_sgd", heads=8, kv_heads=4, inter=2816, layers=8, vocab=32000, tied=False,
              batch=8, seq=384, accum=1, optimizer="sgd", padding="left", positions="sample",
              overlap=False, diagnostics=True),
        # fp16 with loss scaling, 64-wide heads: what the portable executor runs on a GPU
        _case("portable_fp16", heads=8, kv_heads=2, head_dim=64, inter=1536, layers=4, vocab=8192,
              batch=8, seq=256, dtype="fp16"),
    ]


def _spread(rng, low, high):
    """A whole number between low and high, even over its logarithm."""
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    ceiling = 0.9 * max(work(c)["flops"] for c in listed())
    while True:
        portable = rng.random() < 0.1
        head_dim = 64 if portable else 128
        kv = rng.choice([1, 2, 4])
        heads = kv * rng.choice([1, 2, 3, 4, 6, 7])
        hidden = heads * head_dim
        case = dict(
            BASE, heads=heads, kv_heads=kv, head_dim=head_dim,
            inter=8 * round(hidden * rng.uniform(2.0, 6.0) / 8),
            layers=_spread(rng, 1, 12), vocab=8 * _spread(rng, 64, 12000), tied=rng.random() < 0.6,
            accum=rng.choice([1, 2, 2, 3, 4]), seq=_spread(rng, 16, 8192),
            optimizer=rng.choice(["adamw", "adamw", "adamw", "sgd"]),
            padding=rng.choice(["none", "ones", "right", "left"]),
            overlap=rng.random() < 0.75, diagnostics=rng.random() < 0.2,
        )
        case["batch"] = case["accum"] * _spread(rng, 1, 12)
        case["positions"] = {"none": "default", "ones": "row"}.get(case["padding"], "sample")
        if portable:
            case["dtype"] = rng.choice(["fp16", "fp32"])
        tokens = case["batch"] * case["seq"]
        # the dense path keeps S x S scores and fp32 logits: what a user runs there is short
        limit = 4096 if portable else 20000
        if tokens < 64 or tokens > limit or (portable and case["seq"] > 512):
            continue
        if _parameters(case) > 5e8 or work(case)["flops"] > ceiling:
            continue
        return case


# ------------------------------------------------------------------------------------ the work
def _matrix_parameters(case):
    """Weights of one layer that enter a matrix product."""
    hidden = case["heads"] * case["head_dim"]
    kv = case["kv_heads"] * case["head_dim"]
    return hidden * (2 * hidden + 2 * kv) + 3 * hidden * case["inter"]


def _parameters(case):
    hidden = case["heads"] * case["head_dim"]
    head = case["vocab"] * hidden * (1 if case["tied"] else 2)
    vectors = 3 * hidden + 2 * case["kv_heads"] * case["head_dim"]
    return case["layers"] * (_matrix_parameters(case) + vectors) + head + hidden


def work(case):
    hidden = case["heads"] * case["head_dim"]
    tokens = case["batch"] * case["seq"]
    matmul = case["layers"] * _matrix_parameters(case) + case["vocab"] * hidden
    # causal attention: S^2 / 2 scores per head, two products forward and four backward
    attention = 6.0 * case["layers"] * hidden * case["seq"] * tokens
    # read and write of the master weights and optimizer state, one gradient written
    per_parameter = 4 + (24 if case["optimizer"] == "adamw" else 8)
    return {"bytes": float(_parameters(case) * per_parameter + 16 * tokens),
            "flops": 6.0 * matmul * tokens + attention}


def tolerance(case):
    # Measured at the third step, which inherits the first two: gradients of this executor against
    # the torch one at the same precision differ by 0.003 (2 layers) to 0.02 (7 layers) in bf16,
    # those of fp16 against fp32 by 0.001 (4 layers); the roundings of the layers add up as a
    # random walk.  fp32 runs repeat to 2e-7.
    if case["dtype"] == "fp32":
        return {"rel": 1e-5}
    return {"rel": (2e-3 if case["dtype"] == "fp16" else 1.2e-2) * math.sqrt(case["layers"])}


# ------------------------------------------------------------------------------------ the step
def _tokens(case, generator):
    """Token ids with the skew of text: frequency falls with rank (log-uniform ids)."""
    u = torch.rand((case["batch"], case["seq"]), generator=generator, device="cuda")
    ids = torch.exp(u * math.log(case["vocab"])).long() - 1
    return ids.clamp_(0, case["vocab"] - 1)


def _inputs(case, generator):
    ids = _tokens(case, generator)
    batch, seq = ids.shape
    where = torch.arange(seq, device="cuda").unsqueeze(0)
    labels, mask, positions = ids, None, None
    if case["padding"] == "ones":
        mask = torch.ones_like(ids)
    elif case["padding"] != "none":
        length = torch.randint(max(2, seq // 3), seq + 1, (batch, 1), generator=generator, device="cuda")
        mask = (where < length if case["padding"] == "right" else where >= seq - length).long()
        labels = ids.masked_fill(mask == 0, -100)
    if case["positions"] == "row":
        positions = where.clone()
    elif case["positions"] == "sample":
        positions = (mask.cumsum(1) - 1).clamp_(min=0)
    return dict(input_ids=ids, labels=labels, attention_mask=mask, position_ids=positions)


class Session:
    """A model in training and the batch it is trained on."""

    def __init__(self, trainer, inputs):
        self.trainer, self.inputs = trainer, inputs

    def __del__(self):
        # Closed as a program closes it.  The autograd edges of the last step tie the runtime to
        # itself in a way Python's collector cannot see: without emptying it, its arenas would
        # stay on the GPU for the rest of the process.
        runtime = self.trainer.runtime
        runtime.close()
        runtime.__dict__.clear()


def prepare(case, seed):
    gc.collect()      # what earlier sessions left in reference cycles
    torch.manual_seed(seed)
    generator = torch.Generator(device="cuda").manual_seed(seed)
    config = Qwen2ModelConfig(
        vocab_size=case["vocab"], hidden_size=case["heads"] * case["head_dim"],
        intermediate_size=case["inter"], num_hidden_layers=case["layers"],
        num_attention_heads=case["heads"], num_key_value_heads=case["kv_heads"],
        tie_word_embeddings=case["tied"])
    model = Qwen2CausalLM(config, device="cuda")
    overlap = case["overlap"]
    runtime = ShardedRuntime(
        device="cuda:0", reshard_after_forward=True, forward_prefetch=overlap,
        backward_prefetch=overlap, async_grad_rs=overlap,
        communication_policy="stream_ordered" if overlap else "conservative",
        diagnostics_enabled=case["diagnostics"], compute_dtype=case["dtype"]).register(model)
    adamw = case["optimizer"] == "adamw"
    trainer = QwenTrainer(model, runtime, lr=1e-5 if adamw else 1e-2, dtype=case["dtype"],
                          optimizer=case["optimizer"], accumulation_steps=case["accum"])
    return Session(trainer, _inputs(case, generator))


def run(state):
    trainer = state.trainer
    result = trainer.train_step(**state.inputs)
    runtime, optimizer = trainer.runtime, trainer.optimizer
    out = dict(loss=result.loss, valid_tokens=result.valid_tokens,
               parameters=runtime.param_arena, gradients=runtime.grad_arena)
    if hasattr(optimizer, "exp_avg"):
        out.update(exp_avg=optimizer.exp_avg, exp_avg_sq=optimizer.exp_avg_sq)
    return out
