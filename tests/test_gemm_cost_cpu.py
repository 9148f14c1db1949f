"""The choice between the GEMM's small-tile plans and its wide tiles (csrc/gemm_cost.h), as a host program."""
import os
import re
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "train_large_model_from_scratch_b200", "csrc")
PROGRAM = r"""
#include <cstdio>
#include "gemm_cost.h"
using namespace tlm;
static SplitPlan pick(int M, int N, int K, int epi) {           // 148 SMs, contiguous operands, heads of 64
  SplitGemm g{};
  g.M = M; g.N = N; g.K = K; g.epi = epi; g.hd = 64;
  g.a_mn = epi == SPLIT_F32_ACC; g.b_mn = epi == SPLIT_F32_ACC || epi == SPLIT_SWIGLU_BWD;
  g.lda = g.a_mn ? M : K; g.ldb = g.b_mn ? N : K; g.ldc = N;
  const bool pair = M >= 256;
  return split_rule(g, wide_rule(M, N, pair ? 256 : 128, epi == SPLIT_SWIGLU ? 128 : 256, K, pair ? 74 : 148, epi == SPLIT_F32_ACC ? 1 : 0), 148);
}
static_assert(weights_ahead_end(0, 50304) == 384 && weights_ahead_end(128, 512) == 512 && weights_ahead_end(64, 65) == 65 && weights_ahead_end(0, 0) == 0, "");
static_assert(148 * (weights_ahead_end(0, 1 << 30) / 64) * 32768 <= (126 << 20) / 4, "a full chip of 256-wide blocks stays in a quarter of L2");
int main() {
  int M, N, K, epi;
  while (std::scanf("%d %d %d %d", &M, &N, &K, &epi) == 4) { const SplitPlan p = pick(M, N, K, epi); std::printf("%d %d\n", p.bn, p.split); }
}
"""


@pytest.fixture(scope="module")
def picks(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("no host compiler")
    d = tmp_path_factory.mktemp("gemm_cost")
    src, out = str(d / "t.cpp"), str(d / "t")
    with open(src, "w") as f:
        f.write(PROGRAM)
    r = subprocess.run(["g++", "-O2", "-std=c++17", "-I", CSRC, "-o", out, src], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr

    def run(products):
        r = subprocess.run([out], input="\n".join(" ".join(map(str, p)) for p in products), capture_output=True, text=True, timeout=60)
        assert r.returncode == 0, r.stderr
        return [tuple(map(int, line.split())) for line in r.stdout.splitlines()]
    return run


BF16, F32_ACC, HEADS, SWIGLU, SWIGLU_BWD = 0, 1, 3, 4, 5


def test_prompt_products_keep_their_order_of_sums(picks):
    """A plan fixes the order in which a result's fp32 partial sums are added. The projections of 333 rows at hidden 1024: packed
    QKV, output, gate | up, down, LM head."""
    assert picks([(333, 2048, 1024, HEADS), (333, 1024, 1024, BF16), (333, 4096, 1024, SWIGLU), (333, 1024, 4096, BF16),
                  (333, 50304, 1024, BF16)]) == [(64, 1), (64, 2), (0, 0), (128, 4), (0, 0)]


@pytest.mark.parametrize("epi", [BF16, F32_ACC, HEADS, SWIGLU, SWIGLU_BWD])
def test_no_plan_changes_at_a_line_in_the_reduction(picks, epi):
    """Around 100 k-blocks nothing happens in the kernels: products on either side keep their plan."""
    blocks = range(90, 111)
    for M in (64, 128, 256, 333, 512, 768, 1024, 1536, 2048):
        for N in (256, 512, 768, 1024, 1536, 2048, 3072):
            got = picks([(M, N, 64 * b, epi) for b in blocks])
            assert len(set(got)) == 1, (M, N, list(zip(blocks, got)))


@pytest.mark.parametrize("name", ["gemm.cu", "gemm_split.cu"])
def test_weights_are_asked_for_ahead_only_so_far(name):
    """A block's requests ahead of its turn end at `weights_ahead_end` (bounds: the program above) and do not come from thread 0,
    whose own loads would queue behind them."""
    with open(os.path.join(CSRC, name)) as f:
        text = f.read()
    first = text.index("tma_prefetch_2d(&tmB") if name == "gemm_split.cu" else text.index("tma_prefetch_3d(&tmB")
    block = text[text.rindex("if (", 0, text.rindex("M <= ", 0, first)):text.index("griddep_wait();", first)]
    assert "threadIdx.x == 64" in block and len(re.findall(r"tma_prefetch_\dd", block)) == len(re.findall(r"tma_prefetch_\dd", text))
    loops = re.findall(r"for \(int k[b0][^;]*; ([^;]*);", block)
    assert loops == ["k0 < end"] and "weights_ahead_end(" in block
