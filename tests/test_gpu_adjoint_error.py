"""Rounding error of the batched adjoint's accumulators against the single-image adjoint's, for every width of the
interleaved layout: long sums (some 1,100 terms a voxel) against the same sums in 64 bits, put together
from short pieces.

The single-image adjoint splits a voxel's terms over two accumulators (x-dominant and y-dominant LORs). One
accumulator for both doubles the rms rounding error of a sum of n equal-sized terms: n additions at partial sums up
to S, against n / 2 at up to S / 2 twice. The bound of 1.4 lies halfway between (in ratio) equal and doubled."""
import pytest
import torch

pytestmark = pytest.mark.gpu
N, PIECE = 1 << 17, 1 << 11


@pytest.mark.parametrize("images", [2, 3, 8])
@pytest.mark.parametrize("tof,nsigma", [(None, 0.0), ((3.66, 1138.0), 3.0)])
def test_batched_adjoint_rounds_as_the_single_one(cuda_lib, images, tof, nsigma):
    from srf_gb300 import kernels
    shape, center, size = [24, 24, 6], [0.0, 0.0, 0.0], [240.0, 240.0, 60.0]
    g = torch.Generator(device="cuda").manual_seed(3)
    a = torch.rand(N, generator=g, device="cuda") * 6.2831853
    off = (torch.rand(N, 4, generator=g, device="cuda") - 0.5) * torch.tensor([160.0, 160.0, 50.0, 50.0], device="cuda")
    lors = torch.zeros(N, 7, device="cuda")
    lors[:, 0], lors[:, 1], lors[:, 2] = 300 * torch.cos(a), 300 * torch.sin(a), off[:, 2]
    lors[:, 3], lors[:, 4], lors[:, 5] = off[:, 0] - lors[:, 0], off[:, 1] - lors[:, 1], off[:, 3]
    values = torch.rand(images, N, generator=g, device="cuda") + 0.5
    kw = dict(tof=tof, tof_nsigma=nsigma)

    def single(b, rows):
        return kernels.backproject(lors[rows], values[b, rows].contiguous(), shape, center, size, adjoint=True, **kw)

    got = kernels.adjoint_batch(lors, values, shape, center, size, **kw)
    err_batch = err_single = 0.0
    for b in range(images):
        ref = torch.zeros(shape, dtype=torch.float64, device="cuda")
        for k in range(0, N, PIECE):
            ref += single(b, slice(k, k + PIECE)).double()
        err_batch += float((got[b].double() - ref).square().sum())
        err_single += float((single(b, slice(0, N)).double() - ref).square().sum())
    assert err_single > 0 and (err_batch / err_single) ** 0.5 <= 1.4, (err_batch / err_single) ** 0.5
