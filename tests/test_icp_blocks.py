"""The block scheduling of the tracking kernels, on the host: k_icp.cu
compiled with one OS thread per CUDA thread.  Under ThreadSanitizer every
pair of accesses to a block's shared memory that no barrier orders is an
error; two blocks together show what a block that runs out of looks leaves
behind."""
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
        src, n = re.subn(r"constexpr int kIdleLimit = [^;]+;", "constexpr int kIdleLimit = 20;", src)
        assert n == 1
    return src


FLAGS = ["g++", "-std=c++17", "-O1", "-g", "-ffp-contract=off", "-w", "-pthread"]


def _build(tmp, *extra):
    for name in ("k_icp.cu", "vs_internal.cuh"):
        (tmp / name).write_text(_host_source(name))
    flags = FLAGS + list(extra) + ["-I", str(tmp), "-I", EMU, "-I", os.path.join(ROOT, "include"), "-isystem",
                                   os.path.join(CUDA, "include"), '-DEMU_ICP="k_icp.cu"']
    objs = []
    for tag, src in (("a", "icp_block.cpp"), ("b", "icp_block.cpp"), ("main", "icp_main.cpp")):
        objs.append(str(tmp / (tag + ".o")))
        subprocess.run(flags + ["-DEMU_BLOCK=" + tag, "-c", os.path.join(EMU, src), "-o", objs[-1]], check=True)
    subprocess.run(flags + objs + ["-o", str(tmp / "icp_main")], check=True)
    return str(tmp / "icp_main")


@pytest.fixture(scope="module")
def plain(tmp_path_factory):
    return _build(tmp_path_factory.mktemp("icp"))


@pytest.fixture(scope="module")
def checked(tmp_path_factory):
    """the program under ThreadSanitizer"""
    tmp = tmp_path_factory.mktemp("icp_tsan")
    (tmp / "probe.cpp").write_text("int main() { return 0; }\n")
    probe = str(tmp / "probe")
    cmd = FLAGS + ["-fsanitize=thread", str(tmp / "probe.cpp"), "-o", probe]
    if subprocess.run(cmd).returncode or subprocess.run([probe]).returncode:
        pytest.skip("ThreadSanitizer does not run here")
    return _build(tmp, "-fsanitize=thread")


def _run(exe, scenario, mode, listed):
    r = subprocess.run([exe, scenario, str(mode), str(int(listed))], capture_output=True, text=True, timeout=300)
    assert "data race" not in r.stderr, r.stderr[:3000]
    assert r.returncode == 0, r.stderr[:3000]
    return json.loads(r.stdout)


@pytest.mark.parametrize("mode,listed", [(KAHAN, False), (KAHAN, True), (FP64, True)])
def test_shared_memory_is_ordered(checked, mode, listed):
    out = _run(checked, "alone", mode, listed)
    assert [out[f]["tracked"] for f in ("frame", "next")] == [1, 1]


@pytest.mark.parametrize("listed", [False, True])
def test_block_that_runs_out_of_looks_changes_nothing(plain, listed):
    """a block leaves while another holds the iteration's last range: the frame
    ends as it does with that block alone"""
    assert _run(plain, "idle", KAHAN, listed) == _run(plain, "alone", KAHAN, listed)


def test_iteration_that_nobody_ends(plain):
    """its frame is lost, counted and leaves the pose; the next one is tracked
    as if it were the first"""
    alone, out = _run(plain, "alone", KAHAN, False), _run(plain, "stuck", KAHAN, False)
    eye = [float(k % 5 == 0) for k in range(16)]
    assert out["frame"] == dict(tracked=0, failed=1, frame=2, iters=0, count=0, T_gc=eye)
    assert out["next"] == dict(alone["frame"], frame=3)
