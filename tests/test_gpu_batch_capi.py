"""srf_projection_batch and srf_projection_adjoint_batch (separate images; the package itself uses them only for
batches beyond 31-bit offsets) through the C interface, image by image against the oracle, with one layout
and with two. Tolerance 1e-5 relative L2 as for the single-image kernels."""
import numpy as np
import pytest
import torch

from conftest import rel_l2

pytestmark = pytest.mark.gpu
TOL = 1e-5


@pytest.mark.parametrize("images", [1, 3, 8])
@pytest.mark.parametrize("tof,nsigma", [(None, 0.0), ((3.66, 1138.0), 3.0), ((3.66, 1138.0), 0.0)])
@pytest.mark.parametrize("shape,vox,n", [([40, 32, 12], (2.0, 2.25, 2.5), 705), ([130, 36, 7], (1.5, 1.5, 4.0), 33)])
@pytest.mark.parametrize("two", [True, False])
def test_matches_oracle(cuda_lib, oracle, images, tof, nsigma, shape, vox, n, two):
    from srf_gb300._lib import call, f32, f32x3, i32, i32x3, i64, i64x3, ptr, stream_ptr
    from srf_gb300.kernels import _tof_ptr
    center, size = [1.5, -2.0, 0.5], [a * b for a, b in zip(shape, vox)]
    rng = np.random.default_rng(images)
    l = rng.uniform(-150, 150, (n, 7)).astype(np.float32)
    l[:, 6] = rng.normal(0, 40, n)
    l[0] = [-100, -100, -10, 100, 100, 10, 0]     # the non-TOF projector's axis tie
    l[1] = [-50, 0, -200, 50, 0, 200, 5]          # steep
    img = rng.random([images] + shape).astype(np.float32)
    vals = rng.random((images, n)).astype(np.float32) - 0.3
    vals[0, ::3] = 0.0
    dev, v = torch.as_tensor(l).cuda(), torch.as_tensor(vals).cuda()
    nx, ny, nz = shape
    x = torch.as_tensor(img).cuda().permute(0, 3, 2, 1).contiguous()
    y = x.permute(0, 1, 3, 2).contiguous()
    t = tof or (0.0, 0.0)
    head = [ptr(dev), i64(n), i32(7), _tof_ptr(dev) if tof else None, i32(7), f32(t[0]), f32(t[1]), f32(nsigma), i32(images)]
    geo = [i32x3(shape), f32x3(center), f32x3(size)]
    xs, ys = i64x3((1, nx, nx * ny)), i64x3((ny, 1, nx * ny))
    p = torch.full((images, n + 3), 7.0, device="cuda")
    call("srf_projection_batch", *head, i64(nx * ny * nz), ptr(x), xs, ptr(y) if two else None, ys if two else None, *geo, ptr(p),
         i64(n + 3), stream_ptr(dev.device))
    assert bool((p[:, n:] == 7.0).all())
    a, b = torch.zeros_like(x), torch.zeros_like(y)
    call("srf_projection_adjoint_batch", *head, ptr(v), i64(n), ptr(a), i64(nx * ny * nz), xs, ptr(b) if two else None,
         ys if two else None, *geo, stream_ptr(dev.device))
    assert two or not b.any()
    g = (a + b.permute(0, 1, 3, 2)).permute(0, 3, 2, 1).cpu().numpy()
    p = p[:, :n].cpu().numpy()
    kw = dict(tof=True, tof_bin=tof[0], tof_sigma2=tof[1], tof_nsigma=nsigma) if tof else {}
    l = l if tof else np.ascontiguousarray(l[:, :6])
    for k in range(images):
        assert rel_l2(p[k], oracle.projection(img[k], l, shape, center, size, **kw)) <= TOL
        assert rel_l2(g[k], oracle.projection_adjoint(vals[k], l, shape, center, size, **kw)) <= TOL
