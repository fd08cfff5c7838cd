"""What launchers set up once (limits of shared memory, cluster sizes) is set up on every device that a process uses."""

import glob
import os
import re
import shutil
import subprocess

import pytest

_CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "returnn_b200", "csrc")

_MAIN = r"""
#include "per_device.h"
#include <stdio.h>
static int device = 0;
static cudaError_t answer = cudaSuccess;
extern "C" cudaError_t cudaGetDevice(int* d) { *d = device; return answer; }
int main() {
  static RbPerDevice a, b;
  int order[] = {0, 0, 1, 0, 63, 1, 63, 64, 64};
  for (int d : order) {
    device = d;
    printf("%d", a.needed());
    a.done();
  }
  answer = cudaErrorUnknown;
  printf(" %d", a.needed());
  answer = cudaSuccess;
  device = 0;
  printf("%d%d\n", a.needed(), b.needed());
}
"""


def test_flags_are_kept_by_device(tmp_path):
    from returnn_b200.ops import build

    nvcc, gxx = build._nvcc(), shutil.which("g++")
    if not nvcc or not gxx:
        pytest.skip("no compiler")
    (tmp_path / "main.cpp").write_text(_MAIN)
    inc = os.path.join(os.path.dirname(os.path.dirname(nvcc)), "include")
    subprocess.run([gxx, "-std=c++17", "-I", _CSRC, "-I", inc, "-o", str(tmp_path / "main"), str(tmp_path / "main.cpp")], check=True)
    out = subprocess.run([str(tmp_path / "main")], check=True, stdout=subprocess.PIPE).stdout.decode()
    # once for each of the devices 0, 1 and 63; always beyond them and where the device is not known; another flag is another flag
    assert out.split() == ["101010011", "101"]


def test_attributes_are_not_guarded_by_one_flag_per_process():
    for path in glob.glob(os.path.join(_CSRC, "*.cu*")):
        text = open(path).read()
        for m in re.finditer(r"static bool (\w+)(\[\d\])*\s*=", text):
            body = text[m.end(): m.end() + 1500].split("\n}\n")[0]
            assert "cudaFuncSetAttribute" not in body, (os.path.basename(path), m.group(1))
