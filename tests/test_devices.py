"""A process with handles on several devices: a kernel's shared-memory attribute
and the blocks that fit belong to a device. The library's launchers, linked with
a CUDA runtime that launches nothing (tests/cpp/fake_cuda.cpp), ask for both
on each device; a device without cooperative launches, or without room for a
block, takes no phase kernel. Runs without a GPU."""
import os
import subprocess

from conftest import ROOT


def test_launchers_configure_every_device(lvg, tmp_path):
    import lvg_build

    lvg_build.build_cuda()
    objs = [os.path.join(lvg_build.OBJ, f"lvg_{n}.o") for n in ("phase", "aggregate", "move", "kernels")]
    exe = str(tmp_path / "devices_test")
    cpp = os.path.join(ROOT, "tests", "cpp")
    cuda = os.path.join(os.path.dirname(os.path.dirname(os.path.realpath(lvg_build._nvcc()))), "include")
    steps = [[lvg_build._nvcc(), *lvg_build.ARCH, "-std=c++17", "-O1", "--expt-relaxed-constexpr", "-I", lvg_build.CSRC,
              "-I", lvg_build.INCLUDE, "-c", os.path.join(cpp, "devices_test.cu"), "-o", str(tmp_path / "t.o")],
             ["g++", "-std=c++17", "-O1", "-I", cuda, "-c", os.path.join(cpp, "fake_cuda.cpp"), "-o",
              str(tmp_path / "f.o")],
             ["g++", str(tmp_path / "t.o"), str(tmp_path / "f.o"), *objs, "-o", exe, "-lpthread"]]
    for cmd in steps:
        r = subprocess.run(cmd, capture_output=True, text=True)
        assert r.returncode == 0, r.stdout + r.stderr
    run = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert run.returncode == 0, run.stdout + run.stderr
