"""srf_relayout against torch: every pair of source and destination orders, sums of two sources, two
destinations, tile remainders, sliced and expanded sources. Bit-equal (one addition per voxel)."""
import itertools

import pytest
import torch

pytestmark = pytest.mark.gpu
SHAPES = [(1, 1, 1), (16, 16, 16), (17, 5, 33), (64, 64, 16), (3, 40, 15)]


def _view(shape, order, seed):
    perm = {"x": (2, 1, 0), "y": (2, 0, 1), "z": (0, 1, 2)}[order]
    g = torch.Generator(device="cuda").manual_seed(seed)
    t = torch.rand([shape[k] for k in perm], generator=g, device="cuda")
    return t.permute([perm.index(k) for k in range(3)])


@pytest.mark.parametrize("shape", SHAPES)
def test_orders(cuda_lib, shape):
    from srf_gb300 import kernels
    for a, b, c, d in itertools.product("xyz", repeat=4):
        s1, s2 = _view(shape, a, 1), _view(shape, b, 2)
        o1, o2 = kernels._empty_layout(shape, c, s1.device), kernels._empty_layout(shape, d, s1.device)
        kernels._relayout(shape, s1, None, o1)
        assert torch.equal(o1, s1)
        kernels._relayout(shape, s1, s2, o1, o2)
        assert torch.equal(o1, s1 + s2) and torch.equal(o2, s1 + s2)


def test_views(cuda_lib):
    from srf_gb300 import kernels
    big = torch.rand((40, 30, 50), device="cuda")
    for src in (big[3:20, ::2, 5:9], big[:, :, 7:8], torch.rand((1, 30, 1), device="cuda").expand(17, 30, 18)):
        out, out_t = kernels._projector_layouts(src, True)
        assert torch.equal(out, src) and torch.equal(out_t, src)
        assert out.stride(0) == 1 and out_t.stride(1) == 1
