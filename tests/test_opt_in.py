"""The limit of a kernel's shared memory is set on each device it is launched on (opt_in.cuh), and every launcher that keeps in
mind that it has set one keeps it so."""
import os
import re
import shutil
import subprocess

import pytest

KERNELS = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "paged_batch_engine_b200", "csrc", "kernels")

RUNTIME = """
#pragma once
#include <stdio.h>
typedef int cudaError_t;
enum { cudaSuccess = 0, cudaFuncAttributeMaxDynamicSharedMemorySize = 8 };
extern int device, device_error, refuse;
inline cudaError_t cudaGetDevice(int* d) { *d = device; return device_error; }
template <typename K> cudaError_t cudaFuncSetAttribute(K* kernel, int, int bytes) {
  printf("%d:%d:%d ", device, kernel(), bytes);
  return refuse;
}
"""
PROGRAM = """
#include "opt_in.cuh"
int device = 0, device_error = 0, refuse = 0;
int one() { return 1; }
int two() { return 2; }
int main() {
  pbe::OptIn a, b;
  for (int d : {0, 0, 3, 0, 3, 15, 15, 16, 16}) { device = d; if (a(100, one)) return 1; }
  printf("| ");
  device = 3;
  for (int bytes : {90, 120, 100, 120}) if (a(bytes, one)) return 1;
  printf("| ");
  for (int d : {1, 1, 0}) { device = d; if (b(200, one, two)) return 2; }
  printf("| ");
  pbe::OptIn c;
  refuse = 7;
  if (c(300, one) != 7) return 3;          // refused: not kept in mind
  refuse = 0;
  if (c(300, one) || c(300, one)) return 4;
  device_error = 9;
  if (c(300, one) != 9) return 5;
  return 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs a C++ compiler")
def test_on_each_device(tmp_path):
    (tmp_path / "cuda_runtime.h").write_text(RUNTIME)
    (tmp_path / "program.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", f"-I{tmp_path}", f"-I{KERNELS}", str(tmp_path / "program.cpp"), "-o", str(tmp_path / "program")],
                   check=True)
    out = subprocess.run([str(tmp_path / "program")], check=True, capture_output=True, text=True).stdout
    assert out.split() == ["0:1:100", "3:1:100", "15:1:100", "16:1:100", "16:1:100", "|", "3:1:120", "|", "1:1:200", "1:2:200", "0:1:200", "0:2:200", "|",
                           "0:1:300", "0:1:300"]


def test_no_launcher_keeps_it_for_all_devices():
    """Where a limit is set anywhere else it is set before every launch: not under a condition on something static."""
    seen, broken = 0, []
    for file in sorted(os.listdir(KERNELS)):
        if not file.endswith((".cu", ".cuh")) or file == "opt_in.cuh":
            continue
        with open(os.path.join(KERNELS, file)) as f:
            text = re.sub(r"//[^\n]*", "", f.read())
        kept = set(re.findall(r"static (?:bool|int|size_t) (\w+)", text))
        seen += len(re.findall(r"static OptIn", text))
        for found in re.finditer(r"cudaFuncSetAttribute", text):
            # the conditions of the function up to here
            before = text[text.rfind("\n}", 0, found.start()) + 1:found.start()]
            names = {n for c in re.findall(r"if \(([^;{]*)\)", before) for n in re.findall(r"\w+", c)}
            if names & kept:
                broken.append(f"{file}: {sorted(names & kept)}")
    assert seen > 15
    assert not broken, broken
