"""The batched projector and adjoint on interleaved images (widths 2, 4 and 8) against the oracle, one image
at a time: unused places of a voxel, LOR counts around the 32-LOR batches, LORs of more than one
64-slab chunk, axis ties and steep LORs, non-square voxels, image strides other than contiguous, and the
layout kernels at tile remainders.

Tolerance 1e-5 relative L2 as for the single-image kernels: the same visits and weights, summed in
another order."""
import numpy as np
import pytest
import torch

from conftest import rel_l2

pytestmark = pytest.mark.gpu
TOL = 1e-5


def _lors(n, seed):
    rng = np.random.default_rng(seed)
    l = rng.uniform(-150, 150, size=(n, 7)).astype(np.float32)
    l[:, 6] = rng.normal(0, 40, n)
    special = [[-100, -100, -10, 100, 100, 10, 0], [-50, 0, -200, 50, 0, 200, 5], [-3, 0, 0, 4, 1, 0, 0],
               [np.nan, 0, 0, 100, 0, 0, 0], [-120, 30, 5, 10, -5, 2, 30]]
    k = min(n, len(special))
    l[:k] = np.array(special, np.float32)[:k]
    return l


@pytest.mark.parametrize("images", [1, 2, 3, 4, 5, 8])
@pytest.mark.parametrize("tof,nsigma", [(False, 0.0), (True, 3.0), (True, 0.0)])
@pytest.mark.parametrize("shape,vox,n", [([40, 32, 12], (2.0, 2.25, 2.5), 705), ([33, 70, 5], (3.0, 3.0, 3.0), 31), ([130, 36, 7], (1.5, 1.5, 4.0), 64)])
def test_batch_matches_oracle(cuda_lib, oracle, images, tof, nsigma, shape, vox, n):
    from srf_gb300 import kernels
    center, size = [1.5, -2.0, 0.5], [a * b for a, b in zip(shape, vox)]
    lors = _lors(n, images)
    finite = np.isfinite(lors).all(1)
    rng = np.random.default_rng(11)
    img = rng.random([images] + shape).astype(np.float32)
    vals = rng.random((images, n)).astype(np.float32) - 0.3
    vals[0, ::3] = 0.0
    kw = dict(tof=True, tof_bin=3.66, tof_sigma2=1138.0, tof_nsigma=nsigma) if tof else {}
    t = (3.66, 1138.0) if tof else None
    dev = torch.as_tensor(lors if tof else np.ascontiguousarray(lors[:, :6])).cuda()
    x = torch.as_tensor(img).cuda()
    xfast = x.permute(0, 3, 2, 1).contiguous().permute(0, 3, 2, 1)
    p = kernels.project_batch(dev, x, center, size, tof=t, tof_nsigma=nsigma).cpu().numpy()
    q = kernels.project_batch(dev, xfast, center, size, tof=t, tof_nsigma=nsigma).cpu().numpy()
    assert np.array_equal(p, q)
    g = kernels.adjoint_batch(dev, torch.as_tensor(vals).cuda(), shape, center, size, tof=t, tof_nsigma=nsigma).cpu().numpy()
    assert not p[:, ~finite].any()
    for b in range(images):
        assert rel_l2(p[b, finite], oracle.projection(img[b], lors[finite], shape, center, size, **kw)) <= TOL
        assert rel_l2(g[b], oracle.projection_adjoint(vals[b, finite], lors[finite], shape, center, size, **kw)) <= TOL


@pytest.mark.parametrize("images,width", [(2, 2), (3, 4), (4, 4), (6, 8), (8, 8)])
@pytest.mark.parametrize("shape", [(32, 32, 32), (33, 5, 65), (1, 70, 31)])
def test_layouts_round_trip(cuda_lib, images, width, shape):
    from srf_gb300 import _lib, kernels
    x = torch.rand((images,) + shape, device="cuda")
    il, il_t = kernels._interleaved(shape, width, x.device, fill=False)
    if il_t is None:
        il_t = torch.empty((shape[2], shape[0], shape[1], width), device="cuda")
    s = _lib.stream_ptr(x.device)
    _lib.call("srf_interleave", _lib.ptr(x), _lib.i64(x.stride(0)), _lib.i64x3(x.stride()[1:]), _lib.i32(images),
              _lib.i32(width), _lib.i32x3(shape), _lib.ptr(il), _lib.ptr(il_t), s)
    assert torch.equal(il[..., :images], x.permute(3, 2, 1, 0)) and not il[..., images:].any()
    assert torch.equal(il_t[..., :images], x.permute(3, 1, 2, 0)) and not il_t[..., images:].any()
    back = torch.empty_like(x)
    _lib.call("srf_deinterleave", _lib.ptr(il), _lib.ptr(il_t), _lib.i32(images), _lib.i32(width), _lib.i32x3(shape),
              _lib.ptr(back), _lib.i64(back.stride(0)), _lib.i64x3(back.stride()[1:]), s)
    assert torch.equal(back, x + x)
