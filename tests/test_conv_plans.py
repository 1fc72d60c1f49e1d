"""The forward convolution plans every shape its entry point promises: Cin any multiple of 16,
Cout up to 256, whatever the image's size and the output's type; the weight gradient's plans
cover every tile and channel, and no sum in tensor memory is longer than it may be.  On the
CPU; the kernels' results are in test_gpu_conv_wide.py and test_gpu_wgrad_sums.py."""
import os
import subprocess

from conftest import ROOT


def test_every_channel_count_has_a_plan(wrk_lib, tmp_path):
    exe = tmp_path / "conv_plans"
    lib_dir = os.path.dirname(wrk_lib.LIB_PATH)
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", os.path.join(ROOT, "offlinerenderer_b200", "csrc"), "-I",
                    os.path.join(cuda, "include"), os.path.join(ROOT, "tests", "cpp", "conv_plans.cpp"), "-o", str(exe),
                    "-L", lib_dir, "-lwrk", f"-Wl,-rpath,{lib_dir}"], check=True)
    lines = subprocess.run([str(exe)], capture_output=True, text=True, check=True, timeout=120).stdout.splitlines()
    assert lines[-1].startswith("plans 19456 "), lines[-1]
    assert lines[:-1] == [], f"{len(lines) - 1} shapes refused: {lines[:5]}"
