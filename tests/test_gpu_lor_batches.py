"""How LORs are dealt to warps must not show in the results: LOR counts around one LOR, the smallest and
largest batch, one and several rounds of all resident warps. Repeated LORs must project to the same bits
wherever they fall; the first occurrences and the backprojection are held to the oracle (1e-5 relative
L2, as for these kernels everywhere)."""
import numpy as np
import pytest
import torch

from conftest import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 15, 16, 17, 31, 33, 997, 48641, 97280, 97281, 200003, 800001])
@pytest.mark.parametrize("tof", [False, True])
def test_counts(cuda_lib, oracle, n, tof):
    from srf_gb300 import kernels
    from srf_gb300._lib import SRF_RATIO_DIV_NO_NAN
    sh, c, s = [40, 32, 12], [1.5, -2.0, 0.5], [80.0, 72.0, 30.0]
    rng = np.random.default_rng(5)
    u = 997
    base = rng.uniform(-150, 150, (u, 7)).astype(np.float32)
    base[:, [2, 5]] *= 0.3
    base[:, 6] = rng.normal(0, 40, u)
    img = (rng.random(sh) + 0.1).astype(np.float32)
    k = min(n, u)
    idx = np.arange(n) % u
    t = (3.66, 1138.0) if tof else None
    kw = dict(tof=True, tof_bin=3.66, tof_sigma2=1138.0) if tof else {}
    lors = torch.as_tensor(base if tof else base[:, :6].copy()).cuda()[torch.as_tensor(idx).cuda()].contiguous()
    x = torch.as_tensor(img).cuda()
    p = kernels.project(lors, x, c, s, tof=t).cpu().numpy()
    assert np.array_equal(p, p[:k][idx])
    if k > 1:
        assert rel_l2(p[:k], oracle.projection(img, base[:k], sh, c, s, **kw)) <= 1e-5
    # every occurrence of a LOR carries its share: the sum is the unique LORs' backprojection
    count = np.bincount(idx, minlength=u)[:k].astype(np.float64)
    vals = rng.random(u).astype(np.float32)
    share = (vals[:k] / count)[idx].astype(np.float32)
    for adjoint, ref in ((False, oracle.backprojection), (True, oracle.projection_adjoint)):
        b = kernels.backproject(lors, torch.as_tensor(share).cuda(), sh, c, s, tof=t, adjoint=adjoint).cpu().numpy()
        assert rel_l2(b, ref(vals[:k], base[:k], sh, c, s, **kw)) <= 1e-5
    # the fused step: ratio of the projections above
    st = kernels.SubsetState(sh, c, s, x.device, x0=x)
    st.subset(lors, torch.as_tensor(share).cuda(), rule=SRF_RATIO_DIV_NO_NAN, eps=1e-5, tof=t)
    got = (st.bp + st.bp_t).cpu().numpy()
    pr = oracle.projection(img, base[:k], sh, c, s, **kw)
    assert rel_l2(got, oracle.backprojection((vals[:k] / (pr + np.float32(1e-5))).astype(np.float32), base[:k], sh, c, s, **kw)) <= 1e-5
