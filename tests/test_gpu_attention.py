"""tcgen05 flash attention (forward / backward) against an fp32 PyTorch reference."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu

CASES = [(2, 256, 4, 2, 64), (1, 384, 2, 1, 128), (1, 1024, 2, 2, 64), (2, 128, 2, 2, 64), (1, 512, 4, 1, 128),
         (2, 320, 8, 2, 32), (1, 200, 4, 4, 32)]


def _ref(qkv, n_q, n_kv):
    from train_large_model_from_scratch_b200.ops import oracle
    q, k, v = qkv[:, :, :n_q], qkv[:, :, n_q:n_q + n_kv], qkv[:, :, n_q + n_kv:]
    return oracle.attention(q, k, v, causal=True)


@pytest.mark.parametrize("B,T,Hq,Hkv,hd", CASES)
def test_flash_fwd(B, T, Hq, Hkv, hd):
    from train_large_model_from_scratch_b200.ops import native
    torch.manual_seed(0)
    qkv = torch.randn(B, T, Hq + 2 * Hkv, hd, device="cuda").to(torch.bfloat16)
    o, lse = native.flash_attn_fwd(qkv, Hq, Hkv, True)
    native.raise_on_device_status()
    ref = _ref(qkv, Hq, Hkv)
    err = (o.float() - ref).abs().max().item()
    assert err < 2e-2, err
    # logsumexp of the scaled scores
    q = qkv[:, :, :Hq].float().permute(0, 2, 1, 3)
    k = qkv[:, :, Hq:Hq + Hkv].float().permute(0, 2, 1, 3).repeat_interleave(Hq // Hkv, 1)
    s = q @ k.transpose(-1, -2) / math.sqrt(hd)
    s = s.masked_fill(torch.ones(T, T, dtype=torch.bool, device="cuda").triu(1), float("-inf"))
    torch.testing.assert_close(lse, torch.logsumexp(s, -1), rtol=1e-3, atol=2e-3)


@pytest.mark.parametrize("B,T,Hq,Hkv,hd", CASES)
def test_flash_bwd(B, T, Hq, Hkv, hd):
    from train_large_model_from_scratch_b200.ops import native
    torch.manual_seed(1)
    qkv = torch.randn(B, T, Hq + 2 * Hkv, hd, device="cuda").to(torch.bfloat16)
    do = torch.randn(B, T, Hq, hd, device="cuda").to(torch.bfloat16)
    o, lse = native.flash_attn_fwd(qkv, Hq, Hkv, True)
    dqkv = native.flash_attn_bwd(do, qkv, o, lse, Hq, Hkv, True)
    native.raise_on_device_status()
    x = qkv.float().requires_grad_()
    _ref(x, Hq, Hkv).backward(do.float())
    for name, sl in (("dq", slice(0, Hq)), ("dk", slice(Hq, Hq + Hkv)), ("dv", slice(Hq + Hkv, None))):
        a, b = dqkv[:, :, sl].float(), x.grad[:, :, sl]
        rel = ((a - b).norm() / b.norm()).item()
        assert rel < 2e-2, (name, rel)


@pytest.mark.parametrize("B,T,Hq,Hkv,hd", [(2, 256, 4, 2, 64), (1, 384, 2, 1, 128), (2, 320, 8, 2, 32), (1, 200, 4, 4, 64)])
@pytest.mark.parametrize("variant", ["reference", "standard"])
def test_flash_bwd_with_transposed_rope_on_the_way_out(B, T, Hq, Hkv, hd, variant):
    """`rope=(cos, sin)`: dQ and dK come back as gradients of the UN-rotated heads. Oracle: the fp32 autograd
    gradient of the rotated heads pushed through the transposed rotation in fp32."""
    from train_large_model_from_scratch_b200.ops import native, oracle
    torch.manual_seed(3)
    qkv = torch.randn(B, T, Hq + 2 * Hkv, hd, device="cuda").to(torch.bfloat16)
    do = torch.randn(B, T, Hq, hd, device="cuda").to(torch.bfloat16)
    cos, sin = oracle.rope_tables(torch.arange(T, device="cuda"), hd, 10000.0, variant)
    o, lse = native.flash_attn_fwd(qkv, Hq, Hkv, True)
    dqkv = native.flash_attn_bwd(do, qkv, o, lse, Hq, Hkv, True, rope=(cos.contiguous(), sin.contiguous()))
    native.raise_on_device_status()
    x = qkv.float().requires_grad_()
    _ref(x, Hq, Hkv).backward(do.float())
    ref = x.grad.clone()
    ref[:, :, :Hq + Hkv] = oracle.rope_bwd(x.grad[:, :, :Hq + Hkv], cos, sin)
    for name, sl in (("dq", slice(0, Hq)), ("dk", slice(Hq, Hq + Hkv)), ("dv", slice(Hq + Hkv, None))):
        a, b = dqkv[:, :, sl].float(), ref[:, :, sl]
        rel = ((a - b).norm() / b.norm()).item()
        assert rel < 2e-2, (name, rel)


def test_flash_fwd_bwd_at_the_headline_shape():
    """B = 8, T = 4096, 16 query / 8 KV heads of 64 (the benchmark's attention shape: 128 (batch, head) pairs,
    32 KV tiles): the kernels run on the whole batch, the fp32 oracle one batch entry at a time."""
    from train_large_model_from_scratch_b200.ops import native
    B, T, Hq, Hkv, hd = 8, 4096, 16, 8, 64
    torch.manual_seed(4)
    qkv = (torch.randn(B, T, Hq + 2 * Hkv, hd, device="cuda") * 0.7).to(torch.bfloat16)
    do = torch.randn(B, T, Hq, hd, device="cuda").to(torch.bfloat16)
    o, lse = native.flash_attn_fwd(qkv, Hq, Hkv, True)
    dqkv = native.flash_attn_bwd(do, qkv, o, lse, Hq, Hkv, True)
    native.raise_on_device_status()
    for b in (0, 3, 7):
        x = qkv[b:b + 1].float().requires_grad_()
        ref = _ref(x, Hq, Hkv)
        assert (o[b:b + 1].float() - ref).abs().max().item() < 2e-2
        ref.backward(do[b:b + 1].float())
        for name, sl in (("dq", slice(0, Hq)), ("dk", slice(Hq, Hq + Hkv)), ("dv", slice(Hq + Hkv, None))):
            a, g = dqkv[b:b + 1, :, sl].float(), x.grad[:, :, sl]
            rel = ((a - g).norm() / g.norm()).item()
            assert rel < 2e-2, (b, name, rel)
        del x, ref
        torch.cuda.empty_cache()


@pytest.mark.parametrize("group", ["1", "2", "5", "64"])
def test_results_do_not_depend_on_the_block_order(group, monkeypatch):
    """The grids are decoded heavy-first over groups of heads (`csrc/tile_order.h`); any group size, including one that
    leaves a smaller last group (3 x 2 query heads and 3 x 1 KV heads in groups of 2 and 5), must give the same tensors."""
    from train_large_model_from_scratch_b200.ops import native
    torch.manual_seed(5)
    B, T, Hq, Hkv, hd = 3, 640, 2, 1, 64
    qkv = torch.randn(B, T, Hq + 2 * Hkv, hd, device="cuda").to(torch.bfloat16)
    do = torch.randn(B, T, Hq, hd, device="cuda").to(torch.bfloat16)
    o0, lse0 = native.flash_attn_fwd(qkv, Hq, Hkv, True)
    d0 = native.flash_attn_bwd(do, qkv, o0, lse0, Hq, Hkv, True)
    monkeypatch.setenv("TLM_ATTN_FWD_GROUP", group)
    monkeypatch.setenv("TLM_ATTN_BWD_GROUP", group)
    o1, lse1 = native.flash_attn_fwd(qkv, Hq, Hkv, True)
    d1 = native.flash_attn_bwd(do, qkv, o1, lse1, Hq, Hkv, True)
    native.raise_on_device_status()
    assert torch.equal(o0, o1) and torch.equal(lse0, lse1)
    assert torch.equal(d0[:, :, Hq:], d1[:, :, Hq:])                       # dK, dV: one block each, fixed order
    rel = ((d0[:, :, :Hq].float() - d1[:, :, :Hq].float()).norm() / d0[:, :, :Hq].float().norm()).item()
    assert rel < 5e-3, rel                                                 # dQ: fp32 adds from several blocks, any order
    ref = _ref(qkv, Hq, Hkv)
    assert (o1.float() - ref).abs().max().item() < 2e-2


@pytest.mark.parametrize("hd", [32, 64, 128])
@pytest.mark.parametrize("B,T,Hq,Hkv", [(1, 1, 1, 1), (2, 127, 2, 1), (1, 129, 4, 4), (2, 513, 6, 2), (1, 1025, 8, 1), (1, 1025, 1, 1), (3, 1001, 12, 4)])
def test_backward_at_the_edges_of_tiles_and_splits(hd, B, T, Hq, Hkv):
    """Head dim 32 (its own 64-byte-swizzled tiles) and 128 (dQ takes turns with dP in tensor memory, two Q tiles and one dO
    tile in shared memory): one step, first and last steps, several query heads per KV head. Few KV tiles share their steps
    between the CTAs of a cluster (2, 4 or 8 in the later cases; with one query head some CTAs get no step). P and dS are rounded to bf16
    (2^-9) before their products and the results once more, so 1e-2 bounds the relative error of every part."""
    from train_large_model_from_scratch_b200.ops import native
    g = torch.Generator(device="cuda").manual_seed(7)
    qkv = torch.randn(B, T, Hq + 2 * Hkv, hd, device="cuda", generator=g).to(torch.bfloat16)
    do = torch.randn(B, T, Hq, hd, device="cuda", generator=g).to(torch.bfloat16)
    o, lse = native.flash_attn_fwd(qkv, Hq, Hkv, True)
    dqkv = native.flash_attn_bwd(do, qkv, o, lse, Hq, Hkv, True)
    native.raise_on_device_status()
    x = qkv.double().requires_grad_()
    q = x[:, :, :Hq].permute(0, 2, 1, 3)
    k, v = (x[:, :, a:a + Hkv].permute(0, 2, 1, 3).repeat_interleave(Hq // Hkv, 1) for a in (Hq, Hq + Hkv))
    s = (q @ k.transpose(-1, -2) / math.sqrt(hd)).masked_fill(torch.ones(T, T, dtype=torch.bool, device="cuda").triu(1), float("-inf"))
    ref = (torch.softmax(s, -1) @ v).permute(0, 2, 1, 3)
    ref.backward(do.double())
    assert ((o.double() - ref).norm() / ref.norm()).item() < 1e-2
    for name, sl in (("dq", slice(0, Hq)), ("dk", slice(Hq, Hq + Hkv)), ("dv", slice(Hq + Hkv, None))):
        a, b = dqkv[:, :, sl].double(), x.grad[:, :, sl]
        # a single position attends to itself alone: dS is exactly zero up to rounding of dP - delta
        bound = 1e-2 * b.norm().item() if T > 1 or name == "dv" else 1e-2 * do.double().norm().item()
        assert (a - b).norm().item() < bound, (name, (a - b).norm().item(), b.norm().item())


@pytest.mark.parametrize("hd", [32, 64, 128])
@pytest.mark.parametrize("B,T,Hq,Hkv", [(1, 130, 2, 1), (2, 257, 3, 3), (1, 1001, 6, 2)])
def test_backward_with_any_split_of_a_tile(hd, B, T, Hq, Hkv, monkeypatch):
    """1, 2, 4 and 8 CTAs per KV tile, set by hand instead of by the rule (which looks at the chip's SM count): the last tile's
    rows end inside a CTA's share and inside a warp, with 8 CTAs some have no step. Bounds as in the test above."""
    from train_large_model_from_scratch_b200.ops import native
    g = torch.Generator(device="cuda").manual_seed(11)
    qkv = torch.randn(B, T, Hq + 2 * Hkv, hd, device="cuda", generator=g).to(torch.bfloat16)
    do = torch.randn(B, T, Hq, hd, device="cuda", generator=g).to(torch.bfloat16)
    o, lse = native.flash_attn_fwd(qkv, Hq, Hkv, True)
    x = qkv.double().requires_grad_()
    q = x[:, :, :Hq].permute(0, 2, 1, 3)
    k, v = (x[:, :, a:a + Hkv].permute(0, 2, 1, 3).repeat_interleave(Hq // Hkv, 1) for a in (Hq, Hq + Hkv))
    s = (q @ k.transpose(-1, -2) / math.sqrt(hd)).masked_fill(torch.ones(T, T, dtype=torch.bool, device="cuda").triu(1), float("-inf"))
    (torch.softmax(s, -1) @ v).permute(0, 2, 1, 3).backward(do.double())
    for split in (1, 2, 4, 8):
        monkeypatch.setenv("TLM_ATTN_BWD_SPLIT", str(split))
        dqkv = native.flash_attn_bwd(do, qkv, o, lse, Hq, Hkv, True)
        native.raise_on_device_status()
        for name, sl in (("dq", slice(0, Hq)), ("dk", slice(Hq, Hq + Hkv)), ("dv", slice(Hq + Hkv, None))):
            a, b = dqkv[:, :, sl].double(), x.grad[:, :, sl]
            assert ((a - b).norm() / b.norm()).item() < 1e-2, (split, name)


@pytest.mark.parametrize("hd", [32, 64, 128])
@pytest.mark.parametrize("T,n_dst,rows", [(256, 2, 128), (200, 3, 72)])
def test_scatter_forms_into_local_buffers(hd, T, n_dst, rows):
    """The forms that store O, and in the backward dQ / dK / dV, into the sequence owners' tensors, with all owners' tensors on
    this GPU: the same numbers as the packed forms, at the right rows and heads and nowhere else."""
    import ctypes
    from train_large_model_from_scratch_b200.ops import attention_cuda, native, oracle
    B, Hq, Hkv = 2, 4, 2
    g = torch.Generator(device="cuda").manual_seed(13)
    qkv = torch.randn(B, T, Hq + 2 * Hkv, hd, device="cuda", generator=g).to(torch.bfloat16)
    do = torch.randn(B, T, Hq, hd, device="cuda", generator=g).to(torch.bfloat16)
    cos, sin = (t.contiguous() for t in oracle.rope_tables(torch.arange(T, device="cuda"), hd, 10000.0, "reference"))
    o, lse = native.flash_attn_fwd(qkv, Hq, Hkv, True)
    dqkv = native.flash_attn_bwd(do, qkv, o, lse, Hq, Hkv, True, rope=(cos, sin))

    def owners(heads):
        bufs = [torch.full((B, rows, heads, hd), 7.0, dtype=torch.bfloat16, device="cuda") for _ in range(n_dst)]
        return bufs, (ctypes.c_void_p * n_dst)(*[b.data_ptr() for b in bufs])
    bufs, ptrs = owners(Hq + 3)
    o2, lse2 = attention_cuda.fwd_scatter(qkv, Hq, Hkv, ptrs, n_dst, rows, Hq + 3, 2)
    assert torch.equal(o, o2) and torch.equal(lse, lse2)
    got = torch.cat(bufs, dim=1)
    assert torch.equal(got[:, :T, 2:2 + Hq], o) and bool((got[:, T:] == 7.0).all())
    assert bool((got[:, :, :2] == 7.0).all()) and bool((got[:, :, 2 + Hq:] == 7.0).all())
    Ht = 2 * (Hq + 2 * Hkv)                                        # this group's heads among those of two groups
    bufs, ptrs = owners(Ht)
    attention_cuda.bwd_scatter(do, qkv, o, lse, Hq, Hkv, (cos, sin), ptrs, n_dst, rows, Ht, Hq, 2 * Hq + Hkv, 2 * Hq + 3 * Hkv)
    native.raise_on_device_status()
    got = torch.cat(bufs, dim=1)
    assert bool((got[:, T:] == 7.0).all())
    for at, sl in ((Hq, slice(0, Hq)), (2 * Hq + Hkv, slice(Hq, Hq + Hkv)), (2 * Hq + 3 * Hkv, slice(Hq + Hkv, None))):
        a, b = got[:, :T, at:at + (sl.stop or Hq + 2 * Hkv) - sl.start].float(), dqkv[:, :, sl].float()
        # dQ: fp32 adds in any order; dK: rotated before instead of after its rounding to bf16
        assert ((a - b).norm() / b.norm()).item() < 5e-3, at
    others = [h for h in range(Ht) if h not in (*range(Hq, 2 * Hq), *range(2 * Hq + Hkv, 2 * Hq + 2 * Hkv), *range(2 * Hq + 3 * Hkv, Ht))]
    assert bool((got[:, :, others] == 7.0).all())
