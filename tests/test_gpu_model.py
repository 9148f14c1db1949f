"""The GPT on the GPU (bf16 kernels) against the same model on CPU (fp32 oracle path)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _build(device, dtype, **over):
    from train_large_model_from_scratch_b200.models import GPT
    from train_large_model_from_scratch_b200.models.modules.init import clear_init_cache
    from train_large_model_from_scratch_b200.training.config import ModelConfig
    clear_init_cache()
    kw = dict(num_layer=2, hidden_size=256, num_attention_heads=4, num_key_value_heads=2,
              intermediate_size=512, vocab_size=4096, block_size=512)
    kw.update(over)
    return GPT(ModelConfig(**kw), device=device, compute_dtype=dtype)


@pytest.mark.parametrize("heads", [(4, 2), (8, 2)])          # head dim 64, and 32 (the shipped 0.25B model's)
def test_dense_model_matches_cpu_oracle(heads):
    from train_large_model_from_scratch_b200.ops import native
    over = dict(num_attention_heads=heads[0], num_key_value_heads=heads[1])
    gpu = _build("cuda", torch.bfloat16, **over)
    cpu = _build("cpu", torch.float32, **over)
    cpu.dense_buf.params.copy_(gpu.dense_buf.params.float().cpu())       # same (bf16-rounded) weights
    g = torch.Generator().manual_seed(0)
    data = torch.randint(0, 4096, (2, 257), generator=g)
    x, y = data[:, :-1].contiguous(), data[:, 1:].contiguous()
    _, lg, _ = gpu(x.cuda(), y.cuda())
    lg.backward()
    _, lc, _ = cpu(x, y)
    lc.backward()
    native.raise_on_device_status()
    assert abs(lg.item() - lc.item()) < 2e-2, (lg.item(), lc.item())
    gg, gc = gpu.dense_buf.main_grad.cpu(), cpu.dense_buf.main_grad
    cos = torch.nn.functional.cosine_similarity(gg, gc, dim=0).item()
    assert cos > 0.995, cos
    for name, (off, n, _) in cpu.dense_buf.layout.items():
        a, b = gg[off:off + n], gc[off:off + n]
        c = torch.nn.functional.cosine_similarity(a, b, dim=0).item()
        assert c > 0.98, (name, c)


@pytest.mark.parametrize("T,over", [(33, {}), (257, dict(num_attention_heads=8)), (1, {}), (160, dict(num_attention_heads=2, num_key_value_heads=1)),
                                    (300, dict(intermediate_size=520, num_layer=3)), (512, dict(num_layer=1))])
def test_blocks_issued_in_one_call_equal_the_per_op_path(T, over):
    """Without gradients the blocks run as one native call with the same kernels: bit-identical logits and loss. A forward hook
    on a sub-module (which the one call could not run) selects the per-op path and still fires."""
    from train_large_model_from_scratch_b200.ops import native
    model = _build("cuda", torch.bfloat16, **over).eval()
    data = torch.randint(0, 4096, (3, T + 1), generator=torch.Generator().manual_seed(3)).cuda()
    x, y = data[:, :-1].contiguous(), data[:, 1:].contiguous()
    with torch.no_grad():
        assert model._one_call_ok(model.wte(x), T)
        logits, _, _ = model(x)
        _, loss, _ = model(x, y)
        seen = []
        handle = model.blocks[0].mlp.register_forward_hook(lambda *a: seen.append(1))
        logits_ref, _, _ = model(x)
        _, loss_ref, _ = model(x, y)
        handle.remove()
    native.raise_on_device_status()
    assert len(seen) == 2 and torch.equal(logits, logits_ref) and abs(loss.item() - loss_ref.item()) < 1e-5
    logits_grad, _, _ = model(x)                                           # gradients on: per-op path, same values
    assert logits_grad.requires_grad and torch.equal(logits, logits_grad.detach())


def _replace(model, where, seen, monkeypatch):
    """Put a wrapper that counts its calls in one of the places the per-op path goes through."""
    from train_large_model_from_scratch_b200.models.modules.attn import Attention
    from train_large_model_from_scratch_b200.models.modules.norm import LayerNorm
    from train_large_model_from_scratch_b200.ops import attention_cuda, functional as F_ops, native
    owner, name = {"instance add_norm": (model.blocks[1].ln_2, "add_norm"), "instance forward": (model.blocks[1].mlp, "forward"),
                   "class add_norm": (LayerNorm, "add_norm"), "class forward": (Attention, "forward"), "op": (F_ops, "linear"),
                   "kernel": (native, "flash_attn_fwd"), "attention": (attention_cuda, "fwd")}[where]
    stock = getattr(owner, name)

    def wrapper(*args, **kwargs):
        seen.append(where)
        return stock(*args, **kwargs)
    monkeypatch.setattr(owner, name, wrapper)


@pytest.mark.parametrize("where", ["instance add_norm", "instance forward", "class add_norm", "class forward", "op", "kernel", "attention"])
def test_what_a_program_replaced_is_called_without_gradients_too(where, monkeypatch):
    """The one native call knows nothing of a method or an op that the program replaced, on one module, on a class or in the
    op modules: such a program gets the per-op path, which calls the replacement, and the one call again afterwards."""
    from train_large_model_from_scratch_b200.ops import native
    model = _build("cuda", torch.bfloat16).eval()
    x = torch.randint(0, 4096, (2, 64), generator=torch.Generator().manual_seed(5)).cuda()
    seen = []
    with torch.no_grad():
        ref, _, _ = model(x)
        with monkeypatch.context() as m:
            _replace(model, where, seen, m)
            assert not model._one_call_ok(model.wte(x), 64)
            got, _, _ = model(x)
        if not where.startswith("instance"):
            assert model._one_call_ok(model.wte(x), 64)
    native.raise_on_device_status()
    assert seen and torch.equal(got, ref)


def test_forward_mode_tangents_are_not_dropped():
    """The ops have no forward-mode rule and say so; a weight with a tangent must not go into the one call, which would
    return logits without one."""
    import torch.autograd.forward_ad as fwad
    model = _build("cuda", torch.bfloat16).eval()
    x = torch.randint(0, 4096, (2, 64), generator=torch.Generator().manual_seed(6)).cuda()
    with torch.no_grad(), fwad.dual_level():
        w = model.blocks[0].ln_2.weight
        dual = fwad.make_dual(w.detach(), torch.ones_like(w))
        with pytest.raises((NotImplementedError, RuntimeError)):
            torch.func.functional_call(model, {"blocks.0.ln_2.weight": dual}, (x,))


def test_strided_weights_stay_on_the_per_op_path():
    """A projection whose weight is a slice of a wider tensor: the per-op kernels take its row pitch, the one call does not."""
    from train_large_model_from_scratch_b200.ops import native
    model = _build("cuda", torch.bfloat16).eval()
    x = torch.randint(0, 4096, (2, 64), generator=torch.Generator().manual_seed(4)).cuda()
    with torch.no_grad():
        ref, _, _ = model(x)
        w = model.blocks[1].attn.c_proj.weight
        wide = torch.zeros(w.shape[0], w.shape[1] + 64, dtype=w.dtype, device="cuda")
        wide[:, :w.shape[1]] = w
        model.blocks[1].attn.c_proj.weight = torch.nn.Parameter(wide[:, :w.shape[1]])
        assert not model._one_call_ok(model.wte(x), 64)
        got, _, _ = model(x)
    native.raise_on_device_status()
    assert torch.equal(got, ref)


def test_training_reduces_loss_on_fixed_batch():
    from train_large_model_from_scratch_b200.parallel.zero1.distributed_optimizer import FusedAdamW
    model = _build("cuda", torch.bfloat16)
    opt = FusedAdamW([model.dense_buf], lr=2e-3, weight_decay=0.0)
    data = torch.randint(0, 4096, (4, 129), generator=torch.Generator().manual_seed(1)).cuda()
    losses = []
    for _ in range(8):
        opt.zero_grad()
        _, loss, _ = model(data[:, :-1].contiguous(), data[:, 1:].contiguous())
        loss.backward()
        opt.step(grad_clip_value=1.0)
        losses.append(loss.item())
    assert losses[-1] < losses[0] - 0.5, losses


def test_smoke_entry():
    import __graft_entry__
    __graft_entry__.smoke()


def test_moe_model_matches_cpu_oracle():
    from train_large_model_from_scratch_b200.ops import native
    kw = dict(use_moe=True, num_experts=4, num_experts_per_tok=2, moe_intermediate_size=256)
    gpu = _build("cuda", torch.bfloat16, **kw)
    cpu = _build("cpu", torch.float32, **kw)
    cpu.dense_buf.params.copy_(gpu.dense_buf.params.float().cpu())
    cpu.expert_buf.params.copy_(gpu.expert_buf.params.float().cpu())
    data = torch.randint(0, 4096, (2, 257), generator=torch.Generator().manual_seed(3))
    x, y = data[:, :-1].contiguous(), data[:, 1:].contiguous()
    _, lg, _ = gpu(x.cuda(), y.cuda())
    lg.backward()
    _, lc, _ = cpu(x, y)
    lc.backward()
    native.raise_on_device_status()
    assert abs(lg.item() - lc.item()) < 3e-2, (lg.item(), lc.item())
    for a, b in ((gpu.dense_buf, cpu.dense_buf), (gpu.expert_buf, cpu.expert_buf)):
        cos = torch.nn.functional.cosine_similarity(a.main_grad.cpu(), b.main_grad, dim=0).item()
        assert cos > 0.98, cos


def test_lm_head_cross_entropy_is_chunk_invariant(monkeypatch):
    """The fused LM-head + cross-entropy gives the same loss and gradients in one chunk and in several."""
    from train_large_model_from_scratch_b200.ops import functional as Fo
    from train_large_model_from_scratch_b200.ops import native
    data = torch.randint(0, 4096, (2, 257), generator=torch.Generator().manual_seed(3))
    x, y = data[:, :-1].contiguous().cuda(), data[:, 1:].contiguous().cuda()
    out = []
    for chunk in (32768, 192):                       # 512 rows: one chunk, then three (the last one ragged)
        monkeypatch.setattr(Fo._LinearCrossEntropy, "CHUNK_ROWS", chunk)
        m = _build("cuda", torch.bfloat16)
        _, loss, _ = m(x, y)
        loss.backward()
        native.raise_on_device_status()
        out.append((loss.item(), m.dense_buf.main_grad.clone()))
    assert abs(out[0][0] - out[1][0]) < 1e-4, (out[0][0], out[1][0])
    cos = torch.nn.functional.cosine_similarity(out[0][1], out[1][1], dim=0).item()
    assert cos > 0.9999, cos
