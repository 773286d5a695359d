"""What the launch code sets up once per device (csrc/per_device.h), with a stand-in for the CUDA calls: every device of a
process gets its own set-up, once, and one that failed is tried again."""
import pathlib
import re
import shutil
import subprocess

import torch

from snowllm_b200.ops import kernels

CSRC = pathlib.Path(__file__).resolve().parent.parent / "snowllm_b200" / "csrc"

PROGRAM = r"""
#include "per_device.h"
#include <initializer_list>

static std::atomic<int> seen[SNK_MAX_DEVICES];

int main() {
  int made[SNK_MAX_DEVICES + 2] = {0}, value = 0;
  bool fail = false;
  auto call = [&](int device) {
    value = 0;
    return snk_per_device(seen, device, &value, [&](int* n) {
      ++made[device];
      *n = 100 + device;
      return fail ? 7 : 0;
    });
  };
  fail = true;
  if (call(1) != 7 || made[1] != 1) return 1;                       // the error comes back
  fail = false;
  if (call(1) != 0 || made[1] != 2 || value != 101) return 2;       // and is not kept
  for (int device : {0, 1, 0, 1, 3, SNK_MAX_DEVICES - 1, 3})
    if (call(device) != 0 || value != 100 + device) return 3;
  if (made[0] != 1 || made[1] != 2 || made[3] != 1 || made[SNK_MAX_DEVICES - 1] != 1) return 4;
  for (int i = 1; i <= 2; ++i)                                      // past the last one that is kept: made every time
    if (call(SNK_MAX_DEVICES) != 0 || made[SNK_MAX_DEVICES] != i || value != 100 + SNK_MAX_DEVICES) return 5;
  return 0;
}
"""


def test_every_device_is_set_up_once(tmp_path):
    compiler = shutil.which("g++") or shutil.which("c++")
    assert compiler, "the launch code's header needs a C++ compiler to be checked"
    source, program = tmp_path / "check.cpp", tmp_path / "check"
    source.write_text(PROGRAM)
    subprocess.run([compiler, "-std=c++17", "-Wall", "-Werror", f"-I{CSRC}", str(source), "-o", str(program)], check=True)
    assert subprocess.run([str(program)]).returncode == 0


def test_no_launch_code_keeps_a_set_up_for_the_whole_process():
    """A device's SMs and a kernel's limit of shared memory, in the sources: kept per device, or not at all."""
    for source in CSRC.glob("*.cu"):
        text = source.read_text()
        assert not re.search(r"static (int|bool) (sms|configured|set|limit_set)\b", text), source.name


def test_sizes_are_asked_for_on_every_device(monkeypatch):
    """What depends on a device's SMs is kept by the device that it was asked for on."""
    device, asked = [0], []

    def fn(name):
        return lambda *sizes: asked.append((name, device[0], sizes)) or device[0]

    monkeypatch.setattr(kernels, "fn", fn)
    monkeypatch.setattr(torch._C, "_cuda_getDevice", lambda: device[0], raising=False)
    for of in (kernels._conv_step_sizes_ok, kernels._norm_product_sizes_ok, kernels._tc_scratch_bytes):
        asked.clear()
        for device[0] in (0, 1, 0, 1):
            assert of(1, 77, 770, 3) == device[0]
        assert [d for _, d, _ in asked] == [0, 1]
