"""The fused step with truncated windows of three or four groups on images they nearly fill, where LORs that
reach a face go group by group: windows of 81 to 156 slabs around the one-chunk limit of 128, ragged and
non-square images, against the oracle (1e-5 relative L2, as for these kernels everywhere)."""
import numpy as np
import pytest
import torch

from conftest import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,vox", [([120, 96, 40], (2.0, 2.0, 2.0)), ([97, 121, 33], (2.5, 2.5, 1.5)),
                                       ([131, 127, 29], (1.61, 1.61, 2.0)), ([120, 100, 33], (1.5, 1.8, 1.7)),
                                       ([70, 64, 20], (1.3, 1.3, 2.0))])
def test_fused_step(cuda_lib, oracle, shape, vox):
    from srf_gb300 import kernels
    from srf_gb300._lib import SRF_RATIO_DIV_NO_NAN
    size, c = [n * v for n, v in zip(shape, vox)], [0.7, -1.1, 0.4]
    rng = np.random.default_rng(11)
    n = 4001
    lors = np.empty((n, 7), np.float32)
    phi, turn = rng.uniform(0, 2 * np.pi, n), np.pi + rng.uniform(-0.5, 0.5, n)
    for k, a in ((0, phi), (3, phi + turn)):
        lors[:, k], lors[:, k + 1] = 300 * np.cos(a), 300 * np.sin(a)
        lors[:, k + 2] = rng.uniform(-0.7, 0.7, n) * size[2]
    lors[:, 6] = rng.normal(0, 60, n)
    img = (rng.random(shape) + 0.1).astype(np.float32)
    y, add = rng.uniform(0.5, 2, n).astype(np.float32), rng.uniform(0, 5, n).astype(np.float32)
    kw = dict(tof=True, tof_bin=3.66, tof_sigma2=1138.0, tof_nsigma=3.0)
    x = torch.as_tensor(img).cuda()
    st = kernels.SubsetState(shape, c, size, x.device, x0=x)
    st.subset(torch.as_tensor(lors).cuda(), torch.as_tensor(y).cuda(), rule=SRF_RATIO_DIV_NO_NAN, eps=1e-5,
              add=torch.as_tensor(add).cuda(), tof=(3.66, 1138.0), tof_nsigma=3.0)
    got = (st.bp + st.bp_t).cpu().numpy()
    p = oracle.projection(img, lors, shape, c, size, **kw)
    want = oracle.backprojection(y / (p + add + np.float32(1e-5)), lors, shape, c, size, **kw)
    assert rel_l2(got, want) <= 1e-5
