"""Rules of the CUDA sources that no test on a GPU can show to be broken: what a compiler happens to do right today."""
import glob
import os
import re

import train_large_model_from_scratch_b200 as pkg

SRC = os.path.join(os.path.dirname(pkg.__file__), "csrc")


def _source(name):
    with open(os.path.join(SRC, name)) as f:
        return f.read()


def _body(text, start):
    """The braced block that opens at or after `start`."""
    i = text.index("{", start)
    depth, j = 0, i
    while True:
        depth += {"{": 1, "}": -1}.get(text[j], 0)
        j += 1
        if depth == 0:
            return text[i:j]


def test_cluster_barriers_join_their_warp_first():
    """`barrier.cluster.*.aligned` needs all lanes of a warp at the instruction; callers leave loops lane by lane (the rows of
    a sequence's last tile), so the one helper that issues it joins the warp itself, and nobody issues it elsewhere."""
    common = _source("common.cuh")
    body = _body(common, common.index("void cluster_sync_all()"))
    assert body.index("__syncwarp();") < body.index("barrier.cluster.arrive")
    for path in glob.glob(os.path.join(SRC, "*.cu*")):
        text = _source(os.path.basename(path))
        n = len(re.findall(r"barrier\.cluster\.arrive", text))
        assert n == (1 if path.endswith("common.cuh") else 0), path


def test_kernels_that_start_early_read_through_plain_loads():
    """A kernel that calls `griddep_wait` lives from before the kernel in front of it has finished writing. The read-only load
    path (`__ldg`, or what the compiler may make of a `const ... __restrict__` argument) is for memory that nothing writes in a
    kernel's whole life, and a compiler need not keep such loads behind the wait."""
    waiting = 0
    for path in glob.glob(os.path.join(SRC, "*.cu")):
        text = _source(os.path.basename(path))
        for m in re.finditer(r"__global__", text):
            signature, body = text[m.start():text.index("{", m.start())], _body(text, m.start())
            if "griddep_wait();" in body:
                waiting += 1
                assert not re.search(r"const\s+\w+\s*\*\s*__restrict__", signature), signature
                assert "__ldg" not in body and "ld.global.nc" not in body, signature
    assert waiting >= 8
    gemm = _source("gemm.cu")                              # its kernels share one body
    body = _body(gemm, gemm.index("void gemm_body("))
    assert "griddep_wait();" in body and "__ldg" not in body and "ld.global.nc" not in body


def test_no_block_leaves_before_the_wait():
    """`griddep_wait` promises that the kernel in front has ended, and with it those before, because it waited itself. A block that
    leaves early, on an error too, breaks that for its successor."""
    kernels = 0
    for path in glob.glob(os.path.join(SRC, "*.cu")):
        text = _source(os.path.basename(path))
        for m in re.finditer(r"__global__|void gemm_body\(", text):
            body = _body(text, m.start())
            at = body.find("griddep_wait();")
            if at >= 0:
                kernels += 1
                for r in re.finditer(r"\breturn;", body):
                    assert "griddep_wait();" in body[:r.start()], (os.path.basename(path), body[:120])
    assert kernels >= 9


def test_a_width_without_a_kernel_is_an_error():
    """The norms pick their kernel with a `switch` whose every case launches and returns; should a width ever get there
    without a case, the call has to fail instead of reporting a launch that did not happen."""
    text = _source("elementwise.cu")
    switches = [m.end() for m in re.finditer(r"switch \((?:D / 256|sp\.nv)\) \{[^\n]*\}\n#undef TLM_RMS_CASE\n", text)]
    assert len(switches) == 4
    assert all(text[at:].lstrip().startswith("return -4;") for at in switches)


def test_waits_of_single_lanes_stay_in_single_lane_code():
    """A wait that gives up answers lane by lane (one lane may see the phase complete, another the abort flag). In front of
    warp-wide instructions a warp would split there for good, so `mbar_wait` is for the code of one lane, and everything that a
    warp runs together asks `mbar_wait_warp`, whose answer is a vote."""
    common = _source("common.cuh")
    assert "__all_sync(0xffffffffu, mbar_wait<CLUSTER>(" in _body(common, common.index("bool mbar_wait_warp("))
    calls = 0
    for path in sorted(glob.glob(os.path.join(SRC, "*.cu"))):
        text = _source(os.path.basename(path))
        for m in re.finditer(r"\bmbar_wait(?:<\w+>)?\(", text):
            calls += 1
            depth, headers = 0, []
            for i in range(m.start() - 1, -1, -1):
                depth += {"}": 1, "{": -1}.get(text[i], 0)
                if depth < 0:
                    depth = 0
                    headers.append(text[text.rindex("\n", 0, i) + 1:i])
            assert any("lane == 0" in h for h in headers), (os.path.basename(path), text[m.start():text.index("\n", m.start())])
    assert calls >= 4
