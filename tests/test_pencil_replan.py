"""Failing CUDA calls while the pressure solve along grid lines is replanned, on the CPU.

Joining an ensemble replans every variant from a destructor, where an exception would end the process.
The program calls it without a visible device, so its first CUDA call fails.
"""
import os
import subprocess

from ressim_b200 import build

HERE = os.path.dirname(os.path.abspath(__file__))


def test_replanning_without_a_device_returns(tmp_path):
    so = build.build()
    exe = str(tmp_path / "replan_host")
    subprocess.run([os.environ.get("NVCC", "nvcc"), "-std=c++17", "-o", exe,
                    os.path.join(HERE, "native", "replan_host.cu"), "-Xlinker", so,
                    "-Xlinker", "-rpath=" + os.path.dirname(so)], check=True, timeout=300)
    run = subprocess.run([exe], env={**os.environ, "CUDA_VISIBLE_DEVICES": ""}, capture_output=True, text=True,
                         timeout=60)
    assert run.returncode == 0, (run.returncode, run.stdout, run.stderr)
