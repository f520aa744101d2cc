"""The shared-memory limit of a kernel is stated once for every device of a process (csrc/include/msb_launch.hpp against a fake runtime)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA = next((d for d in (os.environ.get("CUDA_HOME"), "/usr/local/cuda") if d and os.path.exists(os.path.join(d, "include", "cuda_runtime_api.h"))), None)

FAKE = r'''
#include "msb_launch.hpp"
#include <cstdio>
static int device = 0, calls = 0, fail = 0;
extern "C" cudaError_t cudaGetDevice(int* d) { *d = device; return cudaSuccess; }
extern "C" cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { ++calls; return fail ? cudaErrorInvalidValue : cudaSuccess; }
extern "C" const char* cudaGetErrorString(cudaError_t) { return "no"; }
extern "C" void msb_set_error(const char*, ...) {}
int main() {
  std::atomic<unsigned long long> stated{0};
  auto at = [&](int d) { device = d; const int rc = msb::allow_smem(nullptr, 1000, "k", stated); printf("%d:%d ", rc, calls); };
  at(0); at(0); at(1); at(1); at(0); at(63); at(63); at(70); at(70);
  fail = 1; at(2); fail = 0; at(2); at(2);
}
'''


@pytest.mark.skipif(CUDA is None or shutil.which("g++") is None, reason="needs the CUDA headers and g++")
def test_every_device_is_told_once(tmp_path):
    src = tmp_path / "fake.cpp"
    src.write_text(FAKE)
    subprocess.run(["g++", "-std=c++17", "-I", os.path.join(ROOT, "mindspeed_b200", "csrc", "include"), "-I", os.path.join(CUDA, "include"),
                    str(src), "-o", str(tmp_path / "fake")], check=True)
    out = subprocess.run([str(tmp_path / "fake")], check=True, capture_output=True, text=True).stdout
    # return code : calls of the runtime so far; a failed statement is made again
    assert out.split() == ["0:1", "0:1", "0:2", "0:2", "0:2", "0:3", "0:3", "0:4", "0:5", "1:6", "0:7", "0:7"]


def test_no_launcher_keeps_a_record_of_its_own():
    """cudaFuncSetAttribute is called in one place."""
    csrc = os.path.join(ROOT, "mindspeed_b200", "csrc")
    named = [f for d, _, fs in os.walk(csrc) for f in fs if f.endswith((".cu", ".cuh", ".hpp", ".cpp"))
             and "cudaFuncSetAttribute" in open(os.path.join(d, f)).read()]
    assert named == ["msb_launch.hpp"]
