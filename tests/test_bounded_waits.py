"""Bounded waits in the kernels' source.  When a wait gives up, some lanes of a warp may and others may not; a warp that goes on
with its lanes' own answers can meet a tcgen05 load, a shuffle or __syncwarp in parts, and then waits for good."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "qllm2_b200", "csrc")

# branches on a wait that one elected thread takes: the producer and the issuer of a GEMM, the issuers of a chunk's products
ONE_THREAD = ["if (!mbar_wait(&empty[", "if (!mbar_wait(&tempty[", "if (!mbar_wait(&full[", "has_s && mbar_wait(&bars[B_DQ]", "has_ds && mbar_wait(&bars[B_DKV]"]


def _lines():
    for name in sorted(os.listdir(CSRC)):
        if name.endswith((".cu", ".cuh")):
            for n, line in enumerate(open(os.path.join(CSRC, name)), 1):
                yield f"{name}:{n}", line.split("//")[0].strip()


def test_branches_on_waits_are_a_warps_or_one_threads():
    branches = [(at, code) for at, code in _lines() if re.search(r"(!|&&|\|\||if \(|while \()\s*(umma::)?mbar_wait\(", code)]
    assert len(branches) == len(ONE_THREAD)
    for at, code in branches:
        assert any(known in code for known in ONE_THREAD), f"{at}: {code}"


def test_stores_by_a_warp_follow_its_common_answer():
    flags = [(at, code) for at, code in _lines() if re.search(r"\bbulk = ", code)]
    assert len(flags) >= 3
    for at, code in flags:
        assert re.search(r"bulk = warp_agrees\(ok\) && \w+\.len == TC;", code), f"{at}: {code}"
