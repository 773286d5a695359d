"""The launch wrappers in C++ (csrc/host.cpp) without a GPU: what they do with tensors that have no memory, and that the entry
points' signatures they are compiled against are the ones that ops/kernels.py declares."""
import pathlib
import re
import subprocess
import sys
import warnings

import pytest

from snowllm_b200.csrc import build
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

NOT_A_NUMBER = """
import ctypes, torch
from torch._subclasses.fake_tensor import FakeTensorMode
from snowllm_b200.csrc import build
host = build.load_host()
NOTHING = ctypes.CFUNCTYPE(ctypes.c_int)(lambda: 0)
SCRATCH = ctypes.CFUNCTYPE(ctypes.c_longlong)(lambda: 64)
for name in ("snk_gemm_simt", "snk_gemm_tc2", "snk_gemm_tc", "snk_add_rmsnorm", "snk_qk_norm_rope_cache", "snk_gemm_tc_parts",
             "snk_moe_topk", "snk_moe_sort"):
    host.bind(name, ctypes.cast(NOTHING, ctypes.c_void_p).value)
host.bind("snk_gemm_tc_scratch_bytes", ctypes.cast(SCRATCH, ctypes.c_void_p).value)
with FakeTensorMode():
    f32 = lambda *s: torch.empty(*s, device="cuda")
    bf = lambda *s: torch.empty(*s, device="cuda", dtype=torch.bfloat16)
    i32 = lambda *s: torch.empty(*s, device="cuda", dtype=torch.int32)
    for out in (host.linear(f32(4, 32), f32(8, 32), 1, 0, None, 3),
                host.linear_add(bf(32, 32), bf(8, 32), f32(32, 8), None, 2),
                host.grouped(bf(32, 32), bf(2, 8, 32), i32(3), None, "1", 1, 0),
                host.add_rmsnorm(f32(4, 32), None, None, None, None, f32(32), "eps", False, None, False),
                host.rope(f32(4, 64), None, None, None, None, 0, i32(4), i32(4), i32(1, 1), 4, f32(1, 2, 1, 4, 16), 2, 1, 16, True),
                host.route_sort(bf(70, 32), bf(8, 32), None, 2, 1, "1", 0, 0)):
        print(out)
"""

LAYOUT_AS_A_NUMBER = """
import ctypes, torch
from torch._subclasses.fake_tensor import FakeTensorMode
from snowllm_b200.csrc import build
host = build.load_host()
host.bind("snk_swiglu", ctypes.cast(ctypes.CFUNCTYPE(ctypes.c_int)(lambda: 0), ctypes.c_void_p).value)
with FakeTensorMode():
    for interleaved in (1, 0, None):
        print(host.swiglu(torch.empty(4, 32, device="cuda"), interleaved))
"""


def run(program: str) -> list:
    done = subprocess.run([sys.executable, "-c", program], cwd=CSRC.parent.parent, capture_output=True, text=True, timeout=300)
    assert done.returncode == 0, done.stderr[-2000:]
    return done.stdout.split()


def test_a_tensor_without_memory_raises():
    """A tensor that has no pointer to give (here one that stands for a CUDA tensor) is an error, and the process goes on."""
    assert run(PROGRAM) == ["raised"] * 6


def test_what_is_no_number_goes_the_long_way():
    """The wrappers in Python say what is wrong with it; these return None for that, and leave no error behind them."""
    assert run(NOT_A_NUMBER) == ["None"] * 6


def test_a_layout_that_is_no_truth_value_goes_the_long_way():
    """Only True meant interleaved columns to the short way, where the wrapper in Python takes any number for one."""
    assert run(LAYOUT_AS_A_NUMBER) == ["None"] * 3


def test_without_the_module_the_wrappers_in_python_do_the_work(monkeypatch):
    """No compiler, or no headers for it: said once, and every call goes the Python wrapper's way."""
    monkeypatch.setattr(kernels, "_native", None)
    monkeypatch.setattr(kernels, "_native_missing", False, raising=False)
    monkeypatch.setattr(build, "_host", None)
    monkeypatch.setattr(build, "host_path", lambda: pathlib.Path("/nowhere/libsnk_host_0.so"))
    monkeypatch.setenv("CXX", "/nowhere/no-such-compiler")
    with pytest.warns(RuntimeWarning, match="wrappers in C\\+\\+"):
        assert kernels.native() is None
    with warnings.catch_warnings():
        warnings.simplefilter("error")
        assert kernels.native() is None
    assert kernels.launch_count() == kernels._launches


def test_another_compiler_or_other_flags_are_another_build(monkeypatch):
    paths = {build.host_path()}
    monkeypatch.setenv("CXX", "some-other-c++")
    paths.add(build.host_path())
    monkeypatch.setattr(build, "HOST_FLAGS", ["-O3"], raising=False)
    paths.add(build.host_path())
    monkeypatch.setattr(build.subprocess, "run", lambda *a, **kw: pytest.fail("ran"))        # a path costs no compiler
    monkeypatch.setattr(build, "_nvcc", lambda: pytest.fail("asked for nvcc"))
    assert build.host_path() in paths and len(paths) == 3


def kinds(arguments: str) -> list:
    """The kinds of a C argument list, as ops/kernels.py has them."""
    out = []
    if arguments.strip() in ("", "void"):
        return out
    for a in re.sub(r"\s+", " ", arguments).split(","):
        a = a.strip()
        if "*" in a or re.match(r"(cudaStream_t|S)\b", a):
            out.append(kernels.P)
        else:
            out.append({"long long": kernels.LL, "int": kernels.I, "float": kernels.F}[re.match(r"(?:const )?(long long|int|float)\b", a)[1]])
    return out


def test_every_entry_point_is_declared_as_it_is_defined():
    """The sources, the table that ctypes goes by, and the types that host.cpp calls through: the same arguments everywhere."""
    defined = {}
    for source in CSRC.glob("*.cu"):
        for name, arguments in re.findall(r"SNK_API (?:int|long long|void) (snk_\w+)\(([^)]*)\)\s*{", source.read_text()):
            defined[name] = kinds(arguments)
    declared = {name: args for table in kernels._SIGNATURES.values() for name, args in table.items()}
    assert len(declared) > 80 and {n: defined.get(n) for n in declared} == declared
    host = (CSRC / "host.cpp").read_text()
    types = {t: kinds(a) for t, a in re.findall(r"typedef (?:int|long long) \(\*(\w+)\)\(([^)]*)\);", host)}
    variables = dict((v, t) for t, v in re.findall(r"^(\w+) (f_\w+);$", host, re.M))
    entries = re.findall(r'{"(snk_\w+)", \(void\*\*\)&(f_\w+)}', host)
    assert len(entries) == len(variables) > 10
    for name, variable in entries:
        assert types[variables[variable]] == declared[name], name
