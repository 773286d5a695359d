"""The launch wrappers in C++ (csrc/host.cpp) without a GPU: what they do with tensors that have no memory, and that the entry
points' signatures they are compiled against are the ones that ops/kernels.py declares."""
import pathlib
import re
import subprocess
import sys

from snowllm_b200.ops import kernels

CSRC = pathlib.Path(kernels.__file__).resolve().parent.parent / "csrc"

PROGRAM = """
import ctypes, torch
from torch._subclasses.fake_tensor import FakeTensorMode
from snowllm_b200.csrc import build
host = build.load_host()
NOTHING = ctypes.CFUNCTYPE(ctypes.c_int)(lambda: 0)
for name in ("snk_swiglu", "snk_add_rmsnorm", "snk_gemm_tc_parts", "snk_gemm_tc_scratch_bytes", "snk_moe_topk", "snk_moe_sort"):
    host.bind(name, ctypes.cast(NOTHING, ctypes.c_void_p).value)
with FakeTensorMode():
    x = torch.empty(4, 32, device="cuda")
    gamma = torch.empty(32, device="cuda")
    for call in (lambda: host.swiglu(x, False), lambda: host.add_rmsnorm(x, None, None, None, None, gamma, 1e-5, False, None, False)):
        for _ in range(3):
            try:
                call()
            except RuntimeError as e:
                print("raised")
"""


def test_a_tensor_without_memory_raises():
    """A tensor that has no pointer to give (here one that stands for a CUDA tensor) is an error, and the process goes on."""
    done = subprocess.run([sys.executable, "-c", PROGRAM], cwd=CSRC.parent.parent, capture_output=True, text=True, timeout=300)
    assert done.returncode == 0, done.stderr[-2000:]
    assert done.stdout.split() == ["raised"] * 6
