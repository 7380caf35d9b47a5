"""The sensitivity image from axial columns against 64 bits: no further off than the line-by-line form, on some of
the clinical scanner's columns (both orders of a pair round independently line by line; the column form
takes one line twice) and on a small scanner's."""
import numpy as np
import pytest
import torch

from conftest import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scanner,columns,shape,vox", [("clinical", 40, [200, 200, 109], (2.04, 2.04, 2.03)),
                                                       ("clinical", 30, [120, 131, 60], (3.4, 2.9, 3.7)),
                                                       ("small", 64, [64, 64, 16], (2.0, 2.0, 2.0))])
@pytest.mark.parametrize("seed", [1, 2])
def test_no_further_from_64_bits_than_line_by_line(cuda_lib, seed, scanner, columns, shape, vox):
    from perf import cases
    from srf_gb300 import ImageConfig, geometry, kernels, synth
    from srf_gb300._lib import call, f32x3, i32, i32x3, i64x3, ptr, stream_ptr
    sc = synth.scanner_clinical() if scanner == "clinical" else synth.scanner_small()
    table = np.asarray(geometry.block_full_crystal_table(sc), np.float32)
    xy, which = np.unique(table[:, :2], axis=0, return_inverse=True)
    pick = np.random.default_rng(seed).permutation(len(xy))[:columns]
    dev = torch.as_tensor(table[np.isin(which.ravel(), pick)]).cuda()
    n, ic = dev.shape[0], ImageConfig(shape, [0.0, 0.0, 0.0], [a * b for a, b in zip(shape, vox)])
    exact = 0.0
    for part in torch.arange(n, device="cuda").split(2000000 // n):
        l = torch.cat([dev[part][:, None].expand(-1, n, 3), dev[None].expand(part.numel(), n, 3)], 2).reshape(-1, 6)
        l = l[(l[:, 3:5] != l[:, :2]).any(1)].contiguous()
        one = torch.ones(l.shape[0], 1, dtype=torch.float64, device="cuda")
        exact = exact + cases._backproject64(one, l, ic, None, 0.0)
    exact = exact.reshape(shape).cpu().numpy()
    a, b = kernels._accumulators(shape, dev.device)
    call("srf_emap_block_full", ptr(dev), i32(1), i32(n), ptr(a), i64x3(a.stride()), ptr(b), i64x3(b.stride()), i32x3(shape),
         f32x3(ic.center), f32x3(ic.size), stream_ptr(dev.device))
    by_line = rel_l2((a + b).cpu().numpy(), exact)
    by_column = rel_l2(kernels.emap_block_full(dev, 1, shape, ic.center, ic.size).cpu().numpy(), exact)
    assert 0 < by_column <= by_line <= 1e-4
