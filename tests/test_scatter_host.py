"""The traversal's scatter (csrc/lean.cuh), compiled for the host and run lane by lane with values 1, infinite
and NaN: it adds value * weight at every slot of non-zero weight and nowhere else. The offsets of slots that
a slab does not visit lie outside the image for many LORs, so an addition that the weight does not decide
is a write out of range."""
import os
import re
import shutil
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "srf_gb300", "csrc")


@pytest.fixture(scope="module")
def scatter_check(tmp_path_factory):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no host compiler")
    d = tmp_path_factory.mktemp("scatter")
    text = '#include "lanes_shim.h"\n'
    for name in ("siddon.cuh", "fused.cuh", "lean.cuh"):
        with open(os.path.join(CSRC, name)) as f:
            s = re.sub(r"#pragma once|#include .*|#pragma unroll", "", f.read())
        text += re.sub(r'asm\("ex2\.approx\.ftz\.f32 %0, %1;" : "=f"\((\w+)\) : "f"\((.*?)\)\);', r"\1 = exp2f(\2);", s)
    with open(os.path.join(HERE, "host", "scatter_check.cpp")) as f:
        text += f.read()
    src = d / "scatter_check.cpp"
    src.write_text(text)
    exe = d / "scatter_check"
    subprocess.run([cxx, "-O2", "-std=c++17", "-ffp-contract=off", "-I", os.path.join(HERE, "host"), str(src), "-o", str(exe)],
                   check=True, capture_output=True, text=True)
    return exe


@pytest.fixture(scope="module")
def lor_file(tmp_path_factory):
    rng = np.random.default_rng(3)
    r = rng.uniform(-150, 150, (4000, 7)).astype(np.float32)
    r[:, [2, 5]] *= 0.2
    r[::7, 3] = -r[::7, 0]
    r[::11, 1] = np.round(r[::11, 1])          # along voxel faces
    r[::11, 4] = r[::11, 1]
    r[::17, 5] *= 8                            # steep
    path = str(tmp_path_factory.mktemp("lors") / "lors")
    r.tofile(path)
    return path


@pytest.mark.parametrize("value", ["1", "inf", "-inf", "nan"])
@pytest.mark.parametrize("tof,nsigma", [(0, 0.0), (1, 0.0), (1, 1.0)])
@pytest.mark.parametrize("grid,size", [((64, 64, 16), (128, 128, 32)), ((41, 37, 9), (128, 100, 32)),
                                       ((110, 90, 30), (210, 168, 60))])
def test_scatter_adds_at_visited_voxels_only(scatter_check, lor_file, value, tof, nsigma, grid, size):
    args = [str(scatter_check), lor_file, *map(str, grid), *map(str, size), str(tof), str(nsigma), value]
    r = subprocess.run(args, check=True, capture_output=True, text=True)
    for line in r.stdout.splitlines():
        n, adds, unvisited, outside, differ = (int(t) for t in line.split())
        assert n > 1000 and adds > 10 * n
        assert unvisited > 1000        # the slots that a wrong decision would write to are there
        assert (outside, differ) == (0, 0), line
