"""The traversal's interior slab code (packed, without range tests; csrc/lean.cuh) against its range-tested form,
compiled for the host: bit-equal weights, equal voxels, offsets inside the image and every slab visited
once, over square, non-square and odd grids, TOF windows and lane counts, for random LORs, LORs through
a scanner's crystals, LORs along voxel faces and at 45 degrees."""
import os
import re
import shutil
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "srf_gb300", "csrc")


@pytest.fixture(scope="module")
def lean_check(tmp_path_factory):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no host compiler")
    d = tmp_path_factory.mktemp("lean")
    text = '#include "device_shim.h"\n'
    for name in ("siddon.cuh", "fused.cuh", "lean.cuh"):
        with open(os.path.join(CSRC, name)) as f:
            s = re.sub(r"#pragma once|#include .*|#pragma unroll", "", f.read())
        # the one inline instruction of these headers: exp2
        text += re.sub(r'asm\("ex2\.approx\.ftz\.f32 %0, %1;" : "=f"\((\w+)\) : "f"\((.*?)\)\);', r"\1 = exp2f(\2);", s)
    with open(os.path.join(HERE, "host", "lean_check.cpp")) as f:
        text += f.read()
    src = d / "lean_check.cpp"
    src.write_text(text)
    exe = d / "lean_check"
    subprocess.run([cxx, "-O2", "-std=c++17", "-ffp-contract=off", "-I", os.path.join(HERE, "host"), str(src), "-o", str(exe)],
                   check=True, capture_output=True, text=True)
    return exe


@pytest.fixture(scope="module")
def lor_files(tmp_path_factory):
    from srf_gb300 import synth
    d = tmp_path_factory.mktemp("lors")
    rng = np.random.default_rng(3)
    r = rng.uniform(-150, 150, (20000, 7)).astype(np.float32)
    r[:, [2, 5]] *= 0.2
    r[::7, 3] = -r[::7, 0]
    r[::11, 1] = np.round(r[::11, 1])          # along voxel faces
    r[::11, 4] = r[::11, 1]
    r[::13, 3:5] = r[::13, 0:2] + np.abs(r[::13, 3:4])  # 45 degrees
    r[::17, 5] *= 8                            # steep
    ic, sc = synth.image_small(), synth.scanner_small()
    e = synth.sample_events(sc, ic, synth.phantom_cylinder(ic), 20000, seed=1, tof_fwhm_ps=530.0).numpy()
    out = {}
    for name, a in (("random", r), ("events", e.astype(np.float32))):
        out[name] = str(d / name)
        a.tofile(out[name])
    return out


@pytest.mark.parametrize("lors", ["random", "events"])
@pytest.mark.parametrize("tof,nsigma", [(0, 0.0), (1, 0.0), (1, 3.0), (1, 0.5)])
@pytest.mark.parametrize("grid,size", [((64, 64, 16), (128, 128, 32)), ((41, 37, 9), (128, 100, 32)),
                                       ((200, 160, 30), (210, 168, 60)), ((33, 70, 50), (99, 196, 20))])
def test_interior_slabs_equal_range_tested(lean_check, lor_files, lors, tof, nsigma, grid, size):
    args = [str(lean_check), lor_files[lors], *map(str, grid), *map(str, size), str(tof), str(nsigma)]
    r = subprocess.run(args, check=True, capture_output=True, text=True)
    for line in r.stdout.splitlines():
        n, hot, slabs, outside, differ, missed = (int(t) for t in line.split())
        assert n > 5000 and slabs > n
        assert (outside, differ, missed) == (0, 0, 0), line
