"""The block scheduling of the tracking kernels, on the host: k_icp.cu
compiled with one OS thread per CUDA thread.  Under ThreadSanitizer every
pair of accesses to a block's shared memory that no barrier orders is an
error."""
import json
import os
import re
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "vcl-volume-scanner_gb300", "csrc")
EMU = os.path.join(ROOT, "tests", "emu")
CUDA = os.path.dirname(os.path.dirname(os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")))
KAHAN, FP64 = 1, 2


def _host_source(name):
    """a kernel file's device code for the host compiler: the two pieces of
    inline PTX as what they compute, and nothing that launches"""
    src = open(os.path.join(CSRC, name)).read()
    src = re.sub(r"asm volatile\(\"bar\.sync 1, 64;\"[^;]*;", "emu_named_barrier();", src)
    src = re.sub(r"asm\(\"rcp\.approx\.ftz\.f(32|64) %0, %1;\"[^;]*\((\w+)\) : \"[fd]\"\((\w+)\)\);",
                 r"\2 = 1.0f / (float)\3;", src)
    assert "asm" not in re.sub(r"//.*", "", src)
    if name == "k_icp.cu":
        src = src[:src.index("void launch_gather_heads(")] + "}  // namespace vs\n"
    return src


@pytest.fixture(scope="module")
def checked(tmp_path_factory):
    """the program under ThreadSanitizer"""
    tmp = tmp_path_factory.mktemp("icp_tsan")
    flags = ["g++", "-std=c++17", "-O1", "-g", "-ffp-contract=off", "-w", "-pthread", "-fsanitize=thread"]
    (tmp / "probe.cpp").write_text("int main() { return 0; }\n")
    probe = str(tmp / "probe")
    if subprocess.run(flags + [str(tmp / "probe.cpp"), "-o", probe]).returncode or subprocess.run([probe]).returncode:
        pytest.skip("ThreadSanitizer does not run here")
    for name in ("k_icp.cu", "vs_internal.cuh"):
        (tmp / name).write_text(_host_source(name))
    flags += ["-I", str(tmp), "-I", EMU, "-I", os.path.join(ROOT, "include"), "-isystem",
              os.path.join(CUDA, "include"), "-DEMU_BLOCK=a", '-DEMU_ICP="k_icp.cu"']
    exe = str(tmp / "icp_main")
    subprocess.run(flags + [os.path.join(EMU, f) for f in ("icp_block.cpp", "icp_main.cpp")] + ["-o", exe],
                   check=True)
    return exe


@pytest.mark.parametrize("mode,listed", [(KAHAN, False), (KAHAN, True), (FP64, True)])
def test_shared_memory_is_ordered(checked, mode, listed):
    r = subprocess.run([checked, str(mode), str(int(listed))], capture_output=True, text=True, timeout=300)
    assert "data race" not in r.stderr, r.stderr[:3000]
    assert r.returncode == 0, r.stderr[:3000]
    out = json.loads(r.stdout)
    assert [out[f]["tracked"] for f in ("frame", "next")] == [1, 1]
