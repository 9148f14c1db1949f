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


# ---------------------------------------------------------------------- backward kernels, against a process that launches one by one
# B, T, query / KV heads, head dim, MLP width, CTAs that share a KV tile (0: the rule's choice). T <= 128 has one KV tile, and dQ
# is one sum; 40 x 128 and 5 x 1000 rows have more than 148 blocks in the pass that also zeroes the dQ accumulator, the others a
# memset. Those two, 1 x 777 and 2 x 500 have small-tile products of 160 to 256 blocks, two to an SM.
BACKWARD = [(3, 100, 8, 2, 32, 520, 0), (2, 128, 4, 4, 64, 512, 0), (40, 128, 4, 2, 64, 1024, 0), (1, 65, 4, 2, 128, 264, 0),
            (1, 777, 8, 2, 64, 1032, 1), (1, 777, 8, 2, 64, 1032, 4), (2, 500, 4, 2, 128, 2048, 2), (5, 1000, 8, 2, 32, 512, 0)]


def _backward_chain(case):
    """Two rounds of a block's forward and backward and of an expert layer's grouped products."""
    import ctypes
    import os
    from train_large_model_from_scratch_b200.ops import native as nat
    B, T, n_q, n_kv, hd, I, split = case
    os.environ.pop("TLM_ATTN_BWD_SPLIT", None)
    if split:
        os.environ["TLM_ATTN_BWD_SPLIT"] = str(split)
    D, Ht, M = n_q * hd, n_q + 2 * n_kv, B * T
    g = torch.Generator(device="cuda").manual_seed(M)
    def rand(*s):
        return torch.randn(*s, generator=g, device="cuda")
    def bf(*s):
        return (rand(*s) * s[-1] ** -0.5).bfloat16()
    wqkv, wo, wgu, wd, nw = bf(Ht * hd, D), bf(D, D), bf(2 * I, D), bf(D, I), torch.ones(D, device="cuda").bfloat16()
    E, counts = 4, [M // 3, 0, M // 2, M - M // 3 - M // 2]
    wp, wde = bf(2 * E, 256, D), bf(E, D, 256)
    ang = torch.arange(T, device="cuda")[:, None] * 10000.0 ** (-torch.arange(0, hd, 2, device="cuda") / hd)
    cos, sin = ang.cos().repeat(1, 2).contiguous(), ang.sin().repeat(1, 2).contiguous()
    cs = nat.rope_table_fp16(cos, sin)
    x, delta, gx = rand(M, D), rand(M, D).bfloat16(), rand(M, D)
    exact, summed, dqs = {}, {}, {}
    acc = {n: torch.zeros(*s, device="cuda") for n, s in
           dict(wqkv=(Ht * hd, D), wo=(D, D), wgu=(2 * I, D), wd=(D, I), norm=(D,), wp=(2 * E, 256, D), wde=(E, D, 256)).items()}
    rs = torch.tensor([0, counts[0], counts[0], counts[0] + counts[2], M], dtype=torch.int32, device="cuda")
    dc = nat.DeviceCounts(rs, max(counts))
    torch.cuda.synchronize()
    for i in range(2):
        x, h, r1 = nat.add_rmsnorm_fwd(x, delta, nw, 1e-5)
        qkv = torch.empty(B, T, Ht, hd, device="cuda", dtype=torch.bfloat16)
        nat.gemm_heads(h, wqkv, False, (ctypes.c_void_p * 1)(qkv.data_ptr()), 1, B, T, T, Ht, 0, n_q, n_kv, n_q, n_kv, hd, n_q + n_kv,
                       cs, 1, (cos, sin))
        o, lse = nat.flash_attn_fwd(qkv, n_q, n_kv, True)
        x2, h2, r2 = nat.add_rmsnorm_fwd(x, nat.gemm_nt(o.view(M, D), wo), nw, 1e-5)
        gu, act = nat.gemm_swiglu(h2, wgu)
        dy = nat.gemm_nt(act, wd)
        dgu = nat.gemm_swiglu_bwd(dy, wd, gu)
        nat.gemm_tn_accum(dy, act, acc["wd"])
        dh2 = nat.gemm_nn(dgu, wgu)
        nat.gemm_tn_accum(dgu, h2, acc["wgu"])
        gx, gd = nat.add_rmsnorm_bwd(gx, dh2, x2, r2, nw, acc["norm"], True)
        do = nat.gemm_nn(gd, wo)
        nat.gemm_tn_accum(gd, o.view(M, D), acc["wo"])
        dqkv = nat.flash_attn_bwd(do.view(B, T, n_q, hd), qkv, o, lse, n_q, n_kv, True, (cos, sin))
        dh = nat.gemm_nn(dqkv.view(M, Ht * hd), wqkv)
        nat.gemm_tn_accum(dqkv.view(M, Ht * hd), h, acc["wqkv"])
        gx1, gd1 = nat.add_rmsnorm_bwd(gx, dh, x, r1, nw, acc["norm"], True)
        egu, eact = nat.grouped_gemm_swiglu(h2, wp, dc)
        ey = nat.grouped_gemm_nt(eact, wde, dc)
        edgu = nat.grouped_gemm_swiglu_bwd(ey, wde, egu, dc)
        nat.grouped_gemm_tn_accum(ey, eact, acc["wde"], dc)
        nat.grouped_gemm_pair_wgrad(edgu, h2, acc["wp"], dc)
        delta = nat.grouped_gemm_pair_dgrad(edgu, wp, dc)
        x = x2
        exact.update({f"{n}{i}": t for n, t in dict(x2=x2, qkv=qkv, o=o, lse=lse, gu=gu, act=act, dgu=dgu, gx=gx, gd=gd, do=do, egu=egu,
                                                    ey=ey, edgu=edgu, delta=delta, dkv=dqkv[:, :, n_q:]).items()})
        (exact if T <= 128 else dqs).update({f"{n}{i}": t for n, t in dict(dq=dqkv[:, :, :n_q], dh=dh, gx1=gx1, gd1=gd1).items()})
    exact["acc_wp"], exact["acc_wde"] = acc.pop("wp"), acc.pop("wde")          # one addition into each of their elements
    dqs.update(acc if T > 128 else {})
    summed.update(acc if T <= 128 else {})
    torch.cuda.synchronize()
    os.environ.pop("TLM_ATTN_BWD_SPLIT", None)
    assert nat.take_device_status() == 0
    return exact, summed, dqs


def _save_backward_chains(path):
    torch.save([tuple({k: v.cpu() for k, v in d.items()} for d in _backward_chain(c)) for c in BACKWARD], path)


@pytest.fixture(scope="module")
def one_by_one(tmp_path_factory):
    """The same calls where every launch waits for its kernel, those inside a call among them."""
    import os
    import subprocess
    import sys
    path = str(tmp_path_factory.mktemp("overlap") / "serial.pt")
    here = os.path.dirname(os.path.abspath(__file__))
    env = dict(os.environ, CUDA_LAUNCH_BLOCKING="1", PYTHONPATH=os.pathsep.join([os.path.dirname(here), here, os.environ.get("PYTHONPATH", "")]))
    r = subprocess.run([sys.executable, "-c", f"import test_gpu_overlap as t; t._save_backward_chains({path!r})"], env=env,
                       capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stdout + r.stderr
    return torch.load(path)


@pytest.mark.parametrize("n", range(len(BACKWARD)))
def test_backward_kernels_are_the_same_one_by_one(one_by_one, n):
    """Bit for bit, but for fp32 sums whose order is open: weight gradients in 2-norm, up to 16 splits or a block per 8 rows of
    terms, 2^-24 sqrt(5120) = 4e-6; dQ with several KV tiles, rounded to bf16 at the end, and what is computed from it: two
    roundings, 2^-8."""
    for _ in range(3):
        for got, ref, tol in zip(_backward_chain(BACKWARD[n]), one_by_one[n], (0.0, 1e-5, 8e-3)):
            assert got.keys() == ref.keys()
            for k in got:
                a, b = got[k].cpu(), ref[k]
                if tol == 0.0:
                    assert torch.equal(a, b), k
                else:
                    assert ((a.double() - b.double()).norm() / b.double().norm()).item() < tol, k
