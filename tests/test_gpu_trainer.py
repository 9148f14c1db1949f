"""The training loop on real GPUs: the recorded (CUDA-graph) step against the ordinary step, and
save -> resume -> loss parity with the recorded step on, at 1 and 2 GPUs."""
import json
import os
import subprocess
import sys
import tempfile

import pytest
import torch

from dist_utils import ROOT, free_port

pytestmark = pytest.mark.gpu

FLAGS = ("--use_mock_data --mock_data_num_samples 256 --seq_len 256 --max_epochs 1 --warmup_steps 4 "
         "--tied_lm_head --num_layer 2 --hidden_size 256 --num_attention_heads 4 --num_key_value_heads 2 "
         "--intermediate_size 512 --vocab_size 8192 --max_lr 1e-3 --min_lr 1e-4 --total_batch_size 4096 "
         "--batch_size 2 --use_distributed_optimizer --sep_size 1").split()


def _run(world, env_extra, flags, log_dir=None):
    if torch.cuda.device_count() < world:
        pytest.skip(f"needs {world} GPUs")
    out = tempfile.mktemp(suffix=".json")
    log_dir = log_dir or tempfile.mkdtemp(prefix="tlm_gpu_")
    env = dict(os.environ, TLM_TEST_OUT=out, PYTHONPATH=ROOT, NCCL_NVLS_ENABLE="0", TLM_NVLS="0")
    env.update(env_extra)
    cmd = [sys.executable, "-m", "torch.distributed.run", "--nnodes=1", f"--nproc-per-node={world}",
           "--master-addr", "127.0.0.1", "--master-port", str(free_port()),
           os.path.join(ROOT, "tests", "_trainer_worker.py")] + flags + ["--log_dir", log_dir]
    r = subprocess.run(cmd, env=env, capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stdout[-3000:] + r.stderr[-3000:]
    with open(out) as f:
        return json.load(f)


def _close(a, b, tol, keys=None):
    for k in (keys if keys is not None else a):
        assert abs(a[k] - b[k]) <= tol * max(1.0, abs(a[k])), (k, a[k], b[k])


@pytest.mark.parametrize("world", [1, 2])
def test_recorded_step_equals_ordinary_step_through_the_warmup_boundary(world):
    """Steps 0-1 run eagerly, step 2 is recorded, steps 3.. replay it; the learning-rate warm-up ends at step
    4, so both schedule branches reach the kernels through the device-side hyper-parameter buffer. Atomic
    reductions (split-K weight gradients, dQ) make the two runs agree to rounding, not bit for bit."""
    eager = _run(world, {"TLM_CUDA_GRAPH": "0"}, FLAGS)
    graph = _run(world, {"TLM_CUDA_GRAPH": "1"}, FLAGS)
    assert len(graph["losses"]) >= 6
    _close(eager["losses"], graph["losses"], 2e-3)
    _close(eager["norms"], graph["norms"], 2e-2)
    assert abs(eager["wsum"] - graph["wsum"]) < 0.5


@pytest.mark.parametrize("world", [1, 2])
def test_save_resume_loss_parity_with_recorded_step(world):
    """An interrupted run (checkpoint at step 4, stop after step 5) continued by a second job must follow
    the uninterrupted run: parameters come back from the fp32 master shards into the (symmetric) bf16 buffer,
    Adam moments and the step counter from the sharded optimizer state, the data position from the sampler."""
    whole = _run(world, {}, FLAGS)
    d = tempfile.mkdtemp(prefix="tlm_gpu_resume_")
    first = _run(world, {"TLM_STOP_AFTER": "6"}, FLAGS + ["--do_save", "--save_every_steps", "4"], log_dir=d)
    assert first["start_step"] == 0
    second = _run(world, {}, FLAGS + ["--do_save", "--save_every_steps", "400"], log_dir=d)
    assert second["start_step"] == 5
    later = [k for k in whole["losses"] if int(k) >= 5]
    assert len(later) >= 3
    _close(whole["losses"], second["losses"], 3e-3, later)
    _close(whole["norms"], second["norms"], 3e-2, later)


def _small_trainer():
    from train_large_model_from_scratch_b200.training import Trainer
    from train_large_model_from_scratch_b200.training.config import (CheckpointConfig, Config, DataConfig, LoggingConfig, ModelConfig,
                                                                     OptimConfig, ParallelConfig, SeedConfig, TrainingConfig)
    return Trainer(Config(
        logging=LoggingConfig(exp_name="t", log_dir=tempfile.mkdtemp(prefix="tlm_gpu_")), seed=SeedConfig(),
        data=DataConfig(use_mock_data=True, mock_data_num_samples=2),
        train=TrainingConfig(total_batch_size=512, batch_size=2, seq_len=256, max_steps=100, max_epochs=None, debug=True).with_derived(),
        optim=OptimConfig(max_lr=6e-4, min_lr=6e-5, warmup_steps=10), ckpt=CheckpointConfig(), parallel=ParallelConfig(),
        model=ModelConfig(num_layer=2, hidden_size=256, num_attention_heads=4, num_key_value_heads=2, intermediate_size=512,
                          vocab_size=2048, block_size=512)))


def test_forward_at_another_length_between_recorded_steps():
    """Scoring a prompt of another length between two steps replaces the rotation tables that the model caches; the recorded
    step goes on reading the ones it was recorded with."""
    data = torch.randint(0, 2048, (2, 257), generator=torch.Generator().manual_seed(8)).cuda()
    batch = [{"input_ids": data[:, :-1].contiguous(), "labels": data[:, 1:].contiguous()}]
    losses = []
    for other_lengths in (False, True):
        tr, run = _small_trainer(), []
        for step in range(7):
            run.append(float(tr.train_step(step, batches=batch)["loss"]))
            if other_lengths and step >= 3:
                logits, _, _ = tr.raw_model(data[:, :100])                 # with gradients on: every block's tables
                del logits
                junk = [torch.full((256, 64), 1e3, device="cuda") for _ in range(64)] + \
                       [torch.full((256, 64, 2), 1e3, device="cuda", dtype=torch.float16) for _ in range(64)]
                del junk
        assert tr._graph is not None
        losses.append(run)
    for a, b in zip(*losses):
        assert abs(a - b) < 5e-3 * a, losses
