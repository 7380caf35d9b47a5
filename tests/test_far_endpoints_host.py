"""LORs whose endpoints lie far outside the image (csrc/fused.cuh, csrc/lean.cuh, compiled for the host): the
rounding of their in-plane coordinates grows with the distance, beyond the margin that keeps the slabs without
range tests inside the image. Whatever the distance, no visited slot may have an offset outside the image."""
import os
import re
import shutil
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "srf_gb300", "csrc")


@pytest.fixture(scope="module")
def range_check(tmp_path_factory):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no host compiler")
    d = tmp_path_factory.mktemp("range")
    text = '#include "device_shim.h"\n'
    for name in ("siddon.cuh", "fused.cuh", "lean.cuh"):
        with open(os.path.join(CSRC, name)) as f:
            s = re.sub(r"#pragma once|#include .*|#pragma unroll", "", f.read())
        text += re.sub(r'asm\("ex2\.approx\.ftz\.f32 %0, %1;" : "=f"\((\w+)\) : "f"\((.*?)\)\);', r"\1 = exp2f(\2);", s)
    with open(os.path.join(HERE, "host", "range_check.cpp")) as f:
        text += f.read()
    src = d / "range_check.cpp"
    src.write_text(text)
    exe = d / "range_check"
    subprocess.run([cxx, "-O2", "-std=c++17", "-ffp-contract=off", "-I", os.path.join(HERE, "host"), str(src), "-o", str(exe)],
                   check=True, capture_output=True, text=True)
    return exe


@pytest.mark.parametrize("distance", [1e3, 1e4, 1e5, 1e6, 1e7, 1e8])
@pytest.mark.parametrize("grid,size", [((64, 64, 16), (128, 128, 32)), ((40, 64, 1), (80, 64, 2)), ((64, 200, 2), (256, 100, 4))])
def test_visited_offsets_are_inside(range_check, tmp_path, distance, grid, size):
    rng = np.random.default_rng(1)
    n = 20000
    half = np.array(size) / 2
    p = rng.uniform(-1, 1, (n, 3)) * half
    # most LORs nearly along an axis and close to the image's faces in the other two
    q = rng.integers(0, 2, n)
    d = np.zeros((n, 3))
    d[np.arange(n), q] = 1.0
    d += rng.uniform(-1, 1, (n, 3)) * 10.0 ** rng.uniform(-9, -1, (n, 1))
    for a in (0, 1, 2):
        vox = size[a] / grid[a]
        near = rng.random(n) < 0.7
        p[near, a] = (rng.choice([-1, 1], n) * (half[a] - vox * 10.0 ** rng.uniform(-4, -0.5, n)))[near]
    lors = np.concatenate([p - distance * d, p + distance * rng.uniform(0.5, 1.5, (n, 1)) * d], 1).astype(np.float32)
    path = str(tmp_path / "lors")
    lors.tofile(path)
    args = [str(range_check), path, *map(str, grid), *map(str, size)]
    n_lors, visits, outside = (int(t) for t in subprocess.run(args, check=True, capture_output=True, text=True).stdout.split())
    assert n_lors > 1000 and visits > n_lors
    assert outside == 0
