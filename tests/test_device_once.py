"""The set-up of kernels per device (csrc/vs_device_once.h), with fake devices."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "vcl-volume-scanner_gb300", "csrc")
CUDA = os.path.dirname(os.path.dirname(os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")))

MAIN = r"""
#include "vs_device_once.h"
#include <cstdio>
#include <thread>
#include <vector>
int main() {
  vs::OncePerDevice once;
  int runs[3] = {0, 0, 0};
  auto set_up = [&](int d, cudaError_t result) { return (int)once.run(d, [&] { runs[d]++; return result; }); };
  printf("%d %d %d ", set_up(0, cudaSuccess), set_up(0, cudaSuccess), set_up(1, cudaSuccess));
  // a failing set-up is reported, and tried again
  printf("%d ", set_up(2, cudaErrorInvalidValue) == (int)cudaErrorInvalidValue);
  printf("%d ", set_up(2, cudaSuccess));
  std::vector<std::thread> ts;
  for (int t = 0; t < 8; t++) ts.emplace_back([&, t] { set_up(t % 3, cudaSuccess); });
  for (auto& t : ts) t.join();
  printf("runs %d %d %d\n", runs[0], runs[1], runs[2]);
}
"""


def test_every_device_is_set_up_once(tmp_path):
    (tmp_path / "main.cpp").write_text(MAIN)
    exe = str(tmp_path / "main")
    subprocess.run(["g++", "-std=c++17", "-pthread", "-I", CSRC, "-isystem", os.path.join(CUDA, "include"),
                    str(tmp_path / "main.cpp"), "-o", exe], check=True)
    assert subprocess.run([exe], capture_output=True, text=True, check=True).stdout == "0 0 0 1 0 runs 1 1 2\n"


def test_sessions_set_kernels_up_on_their_device():
    """no flag of the process stands before the set-up of a session's kernels"""
    src = open(os.path.join(CSRC, "vs_api.cu")).read()
    assert "call_once" not in src and "g_kernels_configured.run(device" in src
