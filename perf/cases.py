"""The workloads whose speed is tracked, from the smallest call to the largest training step.

Four kinds of case, each through the entry points a user's program calls:

  train   `Trainer.train_step`: one whole optimizer step (every micro-step's forward and backward, gradient norm, clip,
          AdamW), bf16, batches resident on the device. What `pretrain_debug.py` does in its loop.
  loss    `GPT(ids, labels)` in evaluation mode without gradients, what `Trainer.eval` does for every validation batch.
  logits  `GPT(ids)`: the full logits of a prompt, what scoring a text with a trained model does.
  moe     one mixture-of-experts layer, forward and backward, as it sits in a GPT block. The layer and not the whole MoE
          model: top-k routing is discrete, so in a deep random-weight model one rounding step before a router sends a
          token to another expert, and two correct builds then differ by more than any tolerance could separate
          from a mistake. With the layer's own input given the routing is reproducible.

Token ids are i.i.d. uniform, weights the framework's own random initialisation, as in its benchmark.
"""
from __future__ import annotations

import math
import tempfile

import torch

from train_large_model_from_scratch_b200.models import GPT
from train_large_model_from_scratch_b200.training import Trainer
from train_large_model_from_scratch_b200.training.config import (CheckpointConfig, Config, DataConfig, LoggingConfig,
                                                                 ModelConfig, OptimConfig, ParallelConfig, SeedConfig,
                                                                 TrainingConfig)

VOCAB = 50304


def _dense(name, kind, layers, hidden, q, kv, inter, seq, batch, accum=1, vocab=VOCAB):
    return dict(name=name, kind=kind, layers=layers, hidden=hidden, q_heads=q, kv_heads=kv, inter=inter, seq=seq,
                batch=batch, accum=accum, vocab=vocab)


def _moe(name, hidden, experts, top_k, inter, seq, batch):
    return dict(name=name, kind="moe", hidden=hidden, experts=experts, top_k=top_k, inter=inter, seq=seq, batch=batch)


def listed():
    return [
        # the plumbing configuration (4 layers of 256, head dim 32): every kernel is a few microseconds, launches and
        # gaps count
        _dense("train_tiny", "train", 4, 256, 8, 2, 1024, 256, 2, accum=2),
        # scripts/debug_gpt_0.25b and example_gpt_0.25b: 12 layers, 32 query / 4 KV heads of dim 32, the shape the
        # launch scripts ship
        _dense("train_shipped_hd32", "train", 12, 1024, 32, 4, 4096, 4096, 8),
        # bench.py's headline configuration: 16 layers, 16 query / 8 KV heads of dim 64, two micro-steps
        _dense("train_headline_hd64", "train", 16, 1024, 16, 8, 4096, 4096, 8, accum=2),
        # the same model on one long sequence (the sequence-parallel configuration's 32768 tokens on one GPU)
        _dense("train_long_32k", "train", 16, 1024, 16, 8, 4096, 32768, 1),
        # bench.py's 3B-class block shape (hidden 3072, 24 query / 8 KV heads of dim 128), six of its layers
        _dense("train_wide_hd128", "train", 6, 3072, 24, 8, 8192, 4096, 2),
        # packed text windows of a length nobody chose for the hardware: odd sequence length, odd batch, an MLP width
        # that is no multiple of 128
        _dense("train_ragged", "train", 8, 768, 12, 4, 2056, 1001, 3, accum=2),
        # validation batches of the headline model
        _dense("eval_headline", "loss", 16, 1024, 16, 8, 4096, 4096, 8),
        # scoring one prompt: latency
        _dense("score_prompt", "logits", 12, 1024, 16, 8, 4096, 333, 1),
        # bench.py's MoE configuration: 8 experts, top 2, expert width 2048, 4 x 4096 tokens
        _moe("moe_8_top2", 1024, 8, 2, 2048, 4096, 4),
        # the MoE defaults of ModelConfig: 128 experts, top 8, expert width 256
        _moe("moe_128_top8", 1024, 128, 8, 256, 2048, 4),
    ]


# ------------------------------------------------------------------------------------------------ drawn cases
def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _odd_sometimes(rng, n, unit):
    """Half of the time a multiple of `unit`, else whatever it is."""
    return max(unit, n // unit * unit) if rng.random() < 0.5 else n


def _draw_once(rng):
    kind = rng.choice(["train", "train", "train", "train", "train", "loss", "logits", "moe", "moe"])
    if kind == "moe":
        experts = rng.choice([4, 8, 16, 32, 64, 128])
        hidden = rng.choice([256, 512, 768, 1024, 1536, 2048])
        inter = rng.choice([128, 256, 512, 768, 1024, 2048])
        tokens = _log_int(rng, 256, 16384)
        batch = rng.randint(1, 4)
        c = _moe("", hidden, experts, rng.choice([1, 2, 2, 4, 8]), inter, _odd_sometimes(rng, max(32, tokens // batch), 128),
                 batch)
        c["top_k"] = min(c["top_k"], experts)
    else:
        head_dim = rng.choice([32, 64, 64, 128])
        hidden = rng.choice([h for h in (256, 512, 768, 1024, 1536, 2048, 3072) if h % head_dim == 0 and h // head_dim <= 64])
        q = hidden // head_dim
        kv = q // rng.choice([r for r in (1, 2, 3, 4, 8) if q % r == 0])
        inter = _odd_sometimes(rng, int(hidden * rng.uniform(2, 4.5)), 128) // 8 * 8
        layers = rng.randint(1, 16)
        vocab = rng.choice([VOCAB, VOCAB, 32000, 8192])
        if kind == "logits":
            seq, batch, accum = _log_int(rng, 16, 4096), 1, 1
        else:
            tokens = _log_int(rng, 256, 32768)
            batch = rng.randint(1, 8)
            seq = _odd_sometimes(rng, max(64, min(32768, tokens // batch)), 128)
            accum = rng.choice([1, 1, 2]) if kind == "train" else 1
        c = _dense("", kind, layers, hidden, q, kv, inter, seq, batch, accum, vocab)
    del c["name"]
    return c


def draw(rng):
    most = max(work(c)["flops"] for c in listed())
    while True:
        c = _draw_once(rng)
        if work(c)["flops"] <= most:
            return c


# ------------------------------------------------------------------------------------------------ states
def _model_config(c) -> ModelConfig:
    return ModelConfig(block_size=max(4096, c["seq"]), vocab_size=c["vocab"], num_layer=c["layers"],
                       num_attention_heads=c["q_heads"], num_key_value_heads=c["kv_heads"], hidden_size=c["hidden"],
                       intermediate_size=c["inter"])


def _tokens(c, seed, n):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    data = torch.randint(0, c["vocab"], (n, c["batch"], c["seq"] + 1), generator=gen, device="cuda")
    return [{"input_ids": d[:, :-1].contiguous(), "labels": d[:, 1:].contiguous()} for d in data]


def _trainer(c) -> Trainer:
    steps = 1_000_000
    cfg = Config(
        logging=LoggingConfig(exp_name="perf", log_dir=tempfile.mkdtemp(prefix="perf_cases_")),
        seed=SeedConfig(),
        data=DataConfig(use_mock_data=True, mock_data_num_samples=c["batch"] * c["accum"]),
        train=TrainingConfig(total_batch_size=c["seq"] * c["batch"] * c["accum"], batch_size=c["batch"], seq_len=c["seq"],
                             max_steps=steps, max_epochs=None, debug=True).with_derived(),
        optim=OptimConfig(max_lr=6e-4, min_lr=6e-5, warmup_steps=1000),
        ckpt=CheckpointConfig(), parallel=ParallelConfig(), model=_model_config(c))
    return Trainer(cfg)


class _TrainState:
    def __init__(self, c, seed):
        self.trainer = _trainer(c)
        self.batches = _tokens(c, seed, c["accum"])
        self.step = 0


class _ForwardState:
    def __init__(self, c, seed):
        self.model = GPT(_model_config(c), device="cuda").eval()
        batch = _tokens(c, seed, 1)[0]
        self.ids = batch["input_ids"]
        self.labels = batch["labels"] if c["kind"] == "loss" else None


class _MoEState:
    def __init__(self, c, seed):
        cfg = ModelConfig(num_layer=1, num_attention_heads=c["hidden"] // 64, num_key_value_heads=c["hidden"] // 64,
                          hidden_size=c["hidden"], vocab_size=256, use_moe=True, num_experts=c["experts"],
                          num_experts_per_tok=c["top_k"], moe_intermediate_size=c["inter"])
        self.model = GPT(cfg, device="cuda")
        self.layer = self.model.blocks[0].mlp
        gen = torch.Generator(device="cuda").manual_seed(seed)
        shape = (c["batch"], c["seq"], c["hidden"])
        # what reaches the layer in a block: RMS-normalised activations, and a loss gradient of a mean over many tokens
        self.x = torch.randn(shape, generator=gen, device="cuda").bfloat16().requires_grad_()
        self.dy = (torch.randn(shape, generator=gen, device="cuda") * 1e-3).bfloat16()


def prepare(case, seed):
    if case["kind"] == "train":
        return _TrainState(case, seed)
    return _MoEState(case, seed) if case["kind"] == "moe" else _ForwardState(case, seed)


def run(s):
    if isinstance(s, _TrainState):
        out = s.trainer.train_step(s.step, batches=s.batches)
        s.step += 1
        flat = s.trainer.raw_model.dense_buf
        return {"loss": out["loss"], "grad_norm": out["grad_norm"], "grads": flat.main_grad, "params": flat.params}
    if isinstance(s, _ForwardState):
        with torch.no_grad():
            logits, loss, _ = s.model(s.ids, s.labels)
        return loss if logits is None else logits
    s.model.zero_grad_buffers()
    s.x.grad = None
    out, logits = s.layer(s.x)
    out.backward(s.dy)
    return {"out": out.detach(), "router_logits": logits.detach(), "dx": s.x.grad, "router_grad": s.layer.router.weight.main_grad,
            "expert_grads": s.model.expert_buf.main_grad}


# ------------------------------------------------------------------------------------------------ what a pass cannot do without
def work(case):
    c = case
    tokens, D, I = c["seq"] * c["batch"], c["hidden"], c["inter"]
    if c["kind"] == "moe":
        E, k = c["experts"], c["top_k"]
        params = 3 * E * D * I + E * D
        # weights read (bf16), their gradients written (fp32); input, output and their gradients (bf16)
        return {"bytes": params * (2 + 4) + tokens * D * 2 * 4, "flops": 3 * (6 * tokens * k * D * I + 2 * tokens * D * E)}
    hd = D // c["q_heads"]
    proj = 2 * D * (c["q_heads"] + 2 * c["kv_heads"]) * hd + 2 * D * D
    layer = tokens * (proj + 6 * D * I)
    attn = 4 * tokens * c["seq"] * D / 2                         # causal: half of the score matrix
    head = 2 * tokens * D * c["vocab"]
    params = c["vocab"] * D + D + c["layers"] * ((c["q_heads"] + 2 * c["kv_heads"]) * hd * D + D * D + 3 * D * I + 2 * D)
    if c["kind"] == "train":
        # backward: twice the forward's products, the score matrix once more. Per parameter: bf16 weight read and
        # written, fp32 master and two moments read and written, fp32 gradient written
        flops = c["accum"] * (3 * c["layers"] * layer + 3.5 * c["layers"] * attn + 3 * head)
        return {"bytes": params * (4 + 24 + 4) + c["accum"] * tokens * 16, "flops": flops}
    out = 4 if c["kind"] == "loss" else tokens * c["vocab"] * 2
    return {"bytes": params * 2 + tokens * (16 if c["kind"] == "loss" else 8) + out, "flops": c["layers"] * (layer + attn) + head}


def tolerance(case):
    # Everything is bf16 between the products, with fp32 accumulation; gradients pass through every layer twice. Measured
    # by running the same step with the library's attention kernels in place of the framework's: gradients differ by
    # 4e-3 (head dim 32 / 64) to 9.6e-3 (six layers of 3072), single ones by up to 0.92 of the root mean square; logits
    # by 3.9e-3 and 0.026; the loss, a mean over many tokens, by 1.5e-6.
    if case["kind"] == "train":
        return {"rel": 2e-2, "max": 0.99}
    if case["kind"] == "loss":
        return {"rel": 2e-5}
    return {"rel": 1.5e-2, "max": 0.4}
