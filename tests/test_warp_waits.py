"""The tcgen05 kernels' waits, in their source: a warp that does more with a barrier than one lane's work waits as one.  A wait for each
lane by itself joins nobody behind it, and what follows (the elected lane's next hand-over, the aligned loads, barriers and
deallocation) takes whole warps; a lane that comes two phases late waits for a phase that never comes."""
import pathlib
import re

import pytest

CSRC = pathlib.Path(__file__).resolve().parent.parent / "snowllm_b200" / "csrc"
WAITS = {"gemm_tc.cu": "mbar_wait", "gemm_tc2.cu": "t2_wait", "attention_tc.cu": "at_wait"}


def block(text: str, at: int) -> str:
    """What stands in the braces that open at or behind ``at``."""
    start = text.index("{", at)
    depth = 0
    for i in range(start, len(text)):
        depth += {"{": 1, "}": -1}.get(text[i], 0)
        if depth == 0:
            return text[start:i + 1]
    raise AssertionError("unbalanced braces")


def kernels(name: str):
    text = re.sub(r"//[^\n]*", "", (CSRC / name).read_text())
    for m in re.finditer(r"__global__ void[^;{]*\bgemm_tc\w*_kernel\(|__global__ void[^;{]*\battention_prefill_tc_kernel\(", text):
        yield block(text, m.end())


@pytest.mark.parametrize("name", WAITS)
def test_a_warp_waits_as_one(name):
    wait = WAITS[name]
    text = (CSRC / name).read_text()
    assert re.search(rf"{wait}_warp\([^)]*\) {{\s*return __all_sync\(0xffffffffu, {wait}\(bar, parity, aborted, code\)\);", text)
    found = list(kernels(name))
    assert len(found) == (2 if name == "gemm_tc2.cu" else 1)
    for body in found:
        issuer = block(body, body.index("} else if (warp == 1) {") + 2)
        rest = body[body.index(issuer) + len(issuer):]                       # the epilogue's warps, and what all warps do at the end
        assert f"{wait}_warp(" in issuer and f"{wait}_warp(" in rest
        for part in (issuer, rest):
            assert not re.search(rf"\b{wait}\(", part)
        # the lane that loads may wait by itself; a wait of the loading warp's lanes together may not
        for line in body[:body.index(issuer)].splitlines():
            assert not re.search(rf"= {wait}\(", line)


@pytest.mark.parametrize("name", WAITS)
def test_warps_are_whole_at_the_end(name):
    for body in kernels(name):
        tail = body[body.rindex("drain_after_abort();"):]
        barrier = tail.index("cluster_sync();") if "cluster_sync();" in tail else tail.index("__syncthreads();")
        assert "__syncwarp();" in tail[:barrier]
        # the aligned barrier of a cluster behind one lane's set-up
        assert all(before.rstrip().endswith("__syncwarp();") for before in body.split("cluster_sync();")[:-1])
