"""Small-tile GEMM: operand rings of every depth, at the edges where a ring fills, wraps and ends in a partial k-block."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bn,split", [(64, 1), (64, 2), (64, 8), (128, 1), (128, 4)])
@pytest.mark.parametrize("blocks", [1, 3, 4, 5, 6, 7, 8, 9, 10, 13, 19, 28])
@pytest.mark.parametrize("kind", ["nt", "nn", "tn"])
def test_rings_of_every_depth(bn, split, blocks, kind):
    from train_large_model_from_scratch_b200.ops import native as nat
    M, N, K = 136, 200, 64 * blocks * split - 24                   # a partial block at the end, for K-major and MN-major operands
    g = torch.Generator(device="cuda").manual_seed(blocks)
    a, b = (torch.randn(r, K, generator=g, device="cuda").bfloat16() for r in (M, N))
    ref = a.double() @ b.double().t()
    am, bm = a.t().contiguous(), b.t().contiguous()
    acc = kind == "tn"
    out = torch.ones(M, N, device="cuda") if acc else torch.empty(M, N, dtype=torch.bfloat16, device="cuda")
    A, lda = (am, M) if kind == "tn" else (a, K)
    B, ldb = (b, K) if kind == "nt" else (bm, N)
    nat._check(nat.lib().tlm_gemm_split(A.data_ptr(), B.data_ptr(), out.data_ptr(), M, N, K, lda, ldb, N, int(kind == "tn"),
                                        int(kind != "nt"), 1 if acc else 0, bn, split, nat._stream()), kind)
    got = out.double() - 1.0 if acc else out.double()
    # fp32 sums of K products (and the ones they are added to); bf16 results are rounded once, 2^-9 relative
    assert ((got - ref).norm() / ref.norm()).item() < (2e-6 if acc else 3e-3)
    assert nat.take_device_status() == 0
