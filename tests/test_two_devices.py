"""The Poisson solve's cluster size is each device's own (a fake of the CUDA
runtime, on the CPU)."""
import os
import shutil
import subprocess

import pytest

from puncpp_gb300 import build_lib

CPP = os.path.join(os.path.dirname(os.path.abspath(__file__)), "cpp")


@pytest.fixture(scope="module")
def exe(lib, tmp_path_factory):
    d = tmp_path_factory.mktemp("devices")
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    main, fake, out = str(d / "main.o"), str(d / "fake.o"), str(d / "two_devices")
    for cmd in ([nvcc] + build_lib.ARCH + build_lib.NVCC_FLAGS + ["-c", os.path.join(CPP, "two_devices.cu"), "-o", main],
                ["g++"] + build_lib.CXX_FLAGS + ["-c", os.path.join(CPP, "fake_cudart.cpp"), "-o", fake],
                ["g++", main, os.path.join(build_lib.BUILD, "k_amg.cu.o"), fake, "-o", out]):
        r = subprocess.run(cmd, capture_output=True, text=True)
        assert r.returncode == 0, r.stderr
    return out


@pytest.mark.parametrize("second", [16, 8])
def test_cluster_size_per_device(exe, second):
    r = subprocess.run([exe] + (["8"] if second == 8 else []), capture_output=True, text=True, timeout=60)
    rows = [tuple(map(int, line.split())) for line in r.stdout.splitlines()]
    # 400 and 12,288 rows on a cluster of 8 and 16 blocks where the device
    # takes them, 12,289 on a grid; the devices in turn, twice
    first, other = [(0, 8), (0, 16), (0, 0)], [(0, 8), (0, second), (0, 0)]
    assert r.returncode == 0 and rows == first + other + first + other
