"""Grouped GEMMs whose workers walk more tiles than one lookup finds (32): where the list is refilled, ends exactly, or ends in a
partly filled batch, for the current tile and for the next one that the epilogue prefetches."""
import random

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(params=["pairs", "single"])
def shape(request):
    """(rows of a tile, workers) of the CTA-pair form and of the single-CTA form."""
    from train_large_model_from_scratch_b200.ops import native as nat
    sms = nat.lib().tlm_num_sms()
    was = nat.set_gemm_pairs(2 if request.param == "pairs" else 0)
    yield (256, sms // 2) if request.param == "pairs" else (128, sms)
    nat.set_gemm_pairs(was)
    assert nat.take_device_status() == 0


def _rand(*s, seed, scale=1.0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return (torch.randn(*s, device="cuda", generator=g) * scale).bfloat16()


def _close(a, b, tol):
    return ((a.float() - b.float()).norm() / b.float().norm()).item() < tol


COLS = 32          # tiles beside each other in a row of tiles


def _groups(tile_rows, workers, per_worker, extra):
    """Ragged and empty groups of `workers * per_worker / COLS` rows of tiles, and `extra` more."""
    rng, left, counts = random.Random(per_worker * 8 + extra), -(-workers * per_worker // COLS) + extra, [0]
    while left > 0:
        tiles = min(left, rng.choice([1, 1, 2, 3, 7, 30]))
        counts.append(tiles * tile_rows - rng.choice([0, 1, 63, tile_rows - 1]))
        counts += [0] * rng.choice([0, 0, 1])
        left -= tiles
    return counts


# 32 tiles for every worker, 33 for some, 64 / 65 for some, more than 64 for all
TOTALS = [(32, 0), (32, 1), (64, 1), (66, 0)]


@pytest.mark.parametrize("per_worker,extra", TOTALS)
def test_row_groups(shape, per_worker, extra):
    """The plain product, gate | up + SwiGLU and its backward; a bf16 result is off by 2^-9 of itself at most."""
    from train_large_model_from_scratch_b200.ops import native as nat
    counts = _groups(*shape, per_worker, extra)
    E, R, K = len(counts), sum(counts), 64
    x = _rand(R + 8, K, seed=1)
    rs = torch.tensor([0] + list(torch.tensor(counts).cumsum(0)), dtype=torch.int32, device="cuda")
    dc = nat.DeviceCounts(rs, max(counts))
    w = _rand(E, COLS * 256, K, seed=2, scale=0.2)
    y = nat.grouped_gemm_nt(x, w, dc)
    wp, I = _rand(2 * E, COLS * 128, K, seed=3, scale=0.2), COLS * 128
    gu, act = nat.grouped_gemm_swiglu(x, wp, dc)
    wd = _rand(E, K, COLS * 256, seed=4, scale=0.2)
    gub = _rand(R + 8, 2 * COLS * 256, seed=5)
    dgu = nat.grouped_gemm_swiglu_bwd(x, wd, gub, dc)
    r = 0
    for e, c in enumerate(counts):
        if c:
            xe = x[r:r + c].float()
            assert _close(y[r:r + c], xe @ w[e].float().t(), 6e-3), ("plain", e)
            g, u = xe @ wp[e].float().t(), xe @ wp[E + e].float().t()
            assert _close(gu[r:r + c, :I], g, 6e-3) and _close(gu[r:r + c, I:], u, 6e-3), ("gate | up", e)
            g, u = gu[r:r + c].float().chunk(2, -1)
            assert _close(act[r:r + c], torch.nn.functional.silu(g) * u, 6e-3), ("swiglu", e)
            dact = (xe @ wd[e].float()).bfloat16().float()
            g, u = gub[r:r + c].float().chunk(2, -1)
            sig = torch.sigmoid(g)
            assert _close(dgu[r:r + c], torch.cat([dact * u * sig * (1 + g * (1 - sig)), dact * g * sig], -1), 8e-3), ("backward", e)
        r += c


@pytest.mark.parametrize("per_worker,extra", TOTALS)
def test_reduction_groups(shape, per_worker, extra):
    """Weight gradients, single and gate | up in one launch: 2048 x 2048 outputs a group, reductions of 0 to 70 rows. fp32 sums."""
    from train_large_model_from_scratch_b200.ops import native as nat
    tile_rows, workers = shape
    N = D = 2048
    E = -(-workers * per_worker // ((N // tile_rows) * (D // 256))) + extra
    counts = [(37 * i) % 71 if i % 5 else 0 for i in range(E)]
    R = sum(counts)
    dy, x = _rand(R + 70, N, seed=6), _rand(R + 70, D, seed=7)
    dy[R:], x[R:] = float("nan"), float("inf")                     # rows behind the last group are not read
    rs = torch.tensor([0] + list(torch.tensor(counts).cumsum(0)), dtype=torch.int32, device="cuda")
    dc = nat.DeviceCounts(rs, R)
    acc = torch.ones(E, N, D, device="cuda")
    nat.grouped_gemm_tn_accum(dy, x, acc, dc)
    acc2 = torch.ones(2 * E, N // 2, D, device="cuda")
    nat.grouped_gemm_pair_wgrad(dy, x, acc2, dc)
    r = 0
    for e, c in enumerate(counts):
        ref = 1.0 + dy[r:r + c].float().t() @ x[r:r + c].float()
        assert _close(acc[e], ref, 1e-4), e
        assert _close(acc2[e], ref[:N // 2], 1e-4) and _close(acc2[E + e], ref[N // 2:], 1e-4), e
        r += c
