"""The LOR setup (csrc/fused.cuh) compiled for the host: its reciprocal division against IEEE division, and
LORs whose TOF value is finite and so large that its quotients by the voxel size and the LOR's length
overflow. Such a value lies infinitely far from the image: every weight is 0, none is NaN."""
import os
import re
import shutil
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "srf_gb300", "csrc")


@pytest.fixture(scope="module")
def setup_check(tmp_path_factory):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no host compiler")
    d = tmp_path_factory.mktemp("setup")
    text = '#include "device_shim.h"\n'
    for name in ("siddon.cuh", "fused.cuh", "lean.cuh"):
        with open(os.path.join(CSRC, name)) as f:
            s = re.sub(r"#pragma once|#include .*|#pragma unroll", "", f.read())
        text += re.sub(r'asm\("ex2\.approx\.ftz\.f32 %0, %1;" : "=f"\((\w+)\) : "f"\((.*?)\)\);', r"\1 = exp2f(\2);", s)
    with open(os.path.join(HERE, "host", "setup_check.cpp")) as f:
        text += f.read()
    src = d / "setup_check.cpp"
    src.write_text(text)
    exe = d / "setup_check"
    subprocess.run([cxx, "-O2", "-std=c++17", "-ffp-contract=off", "-I", os.path.join(HERE, "host"), str(src), "-o", str(exe)],
                   check=True, capture_output=True, text=True)
    return exe


@pytest.mark.parametrize("seed", [1, 2])
def test_division_is_ieee(setup_check, seed):
    r = subprocess.run([str(setup_check), "division", "4000000", str(seed)], check=True, capture_output=True, text=True)
    n, differ = (int(t) for t in r.stdout.split())
    assert n == 4000000 and differ == 0


@pytest.mark.parametrize("value", [3.4e38, -3.4e38, 1e38, -1.7e38, 1e30])
@pytest.mark.parametrize("nsigma", [0.0, 3.0])
@pytest.mark.parametrize("grid,size", [((64, 64, 16), (32, 32, 8)), ((41, 37, 9), (20, 15, 4)), ((64, 64, 16), (128, 128, 32))])
def test_overflowing_tof_values(setup_check, tmp_path, value, nsigma, grid, size):
    rng = np.random.default_rng(7)
    l = rng.uniform(-1.5, 1.5, (500, 7)).astype(np.float32) * (np.float32(size[0]))
    l[:, [2, 5]] *= 0.1
    l[:, 6] = value
    path = str(tmp_path / "lors")
    l.tofile(path)
    args = [str(setup_check), "tof", path, *map(str, grid), *map(str, size), str(nsigma)]
    n, slabs, nan, nonzero = (int(t) for t in subprocess.run(args, check=True, capture_output=True, text=True).stdout.split())
    assert n == 500 and (nan, nonzero) == (0, 0)
    assert nsigma > 0 or slabs > 500  # untruncated LORs are walked
