"""Kernels that start before the one in front of them is done give what they give one at a time, bit for bit."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _chain(nat, T, D, n_q, n_kv, I, layers, sync):
    """Blocks' forward and backward kernels in a row, buffers taken from and given back to the allocator on the way."""
    g = torch.Generator(device="cuda").manual_seed(T)
    def bf(*s):
        return (torch.randn(*s, generator=g, device="cuda") * s[-1] ** -0.5).bfloat16()
    hd = D // n_q
    wqkv, wo, wgu, wd, nw = bf((n_q + 2 * n_kv) * hd, D), bf(D, D), bf(2 * I, D), bf(D, I), torch.ones(D, device="cuda").bfloat16()
    wait = torch.cuda.synchronize if sync else (lambda: None)
    x, delta, out = torch.randn(T, D, generator=g, device="cuda"), None, []
    for _ in range(layers):
        x, h, rstd = nat.add_rmsnorm_fwd(x, delta, nw, 1e-5); wait()
        qkv = nat.gemm_nt(h, wqkv).view(1, T, n_q + 2 * n_kv, hd); wait()
        o, lse = nat.flash_attn_fwd(qkv, n_q, n_kv, True); wait()
        a = nat.gemm_nt(o.view(T, D), wo); wait()
        x, h, rstd = nat.add_rmsnorm_fwd(x, a, nw, 1e-5); wait()
        gu, act = nat.gemm_swiglu(h, wgu); wait()
        delta = nat.gemm_nt(act, wd); wait()
        dgu = nat.gemm_swiglu_bwd(delta, wd, gu); wait()
        dh = nat.gemm_nn(dgu, wgu); wait()
        do = nat.gemm_nn(dh, wo).view(1, T, n_q, hd); wait()
        out += [qkv, lse, act, dgu, do]
    out += [x, delta]
    torch.cuda.synchronize()
    return out


@pytest.mark.parametrize("T,D,n_q,n_kv,I", [(1, 256, 4, 2, 512), (33, 256, 8, 2, 264), (333, 1024, 16, 8, 4096), (512, 256, 8, 2, 1024),
                                            (1003, 768, 12, 4, 2056), (1280, 512, 4, 4, 1024)])
def test_a_chain_of_kernels_is_the_same_with_and_without_waiting(T, D, n_q, n_kv, I):
    from train_large_model_from_scratch_b200.ops import native as nat
    one_by_one = _chain(nat, T, D, n_q, n_kv, I, 4, True)
    for _ in range(3):
        for a, b in zip(_chain(nat, T, D, n_q, n_kv, I, 4, False), one_by_one):
            assert torch.equal(a, b)
    assert nat.take_device_status() == 0
