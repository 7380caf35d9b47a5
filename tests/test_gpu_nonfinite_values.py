"""LOR values that are infinite or NaN, on the kernels that scatter by slot (csrc/lean.cuh): they reach the
voxels that their LORs visit and nothing else. The accumulators stand inside a larger buffer whose margins
must stay untouched (tests/test_scatter_host.py shows the addresses without a GPU).

Tolerance 1e-5 relative L2 where two sums of the same terms in another order are compared."""
import numpy as np
import pytest
import torch

from conftest import rel_l2

pytestmark = pytest.mark.gpu
TOL = 1e-5
MARGIN = 1 << 18
TOF = (3.66, 1138.0)
BAD = [np.nan, np.inf, -np.inf]


def _lors(n, seed):
    """Random LORs, most of them through the image's faces and some beside it."""
    rng = np.random.default_rng(seed)
    l = rng.uniform(-150, 150, (n, 7)).astype(np.float32)
    l[:, [2, 5]] *= 0.3
    l[:, 6] = rng.normal(0, 40, n)
    l[::5, [1, 4]] = rng.uniform(140, 150, (len(l[::5]), 2))   # beside the image
    l[::17, 5] *= 5
    return torch.as_tensor(l).cuda()


def _padded(shape):
    """x-fastest and y-fastest accumulators with margins on both sides, and the margins."""
    nx, ny, nz = shape
    v = nx * ny * nz
    buf = torch.zeros(2 * v + 3 * MARGIN, device="cuda")
    a, b = buf[MARGIN:MARGIN + v], buf[2 * MARGIN + v:2 * MARGIN + 2 * v]
    rims = [buf[:MARGIN], buf[MARGIN + v:2 * MARGIN + v], buf[2 * MARGIN + 2 * v:]]
    return a.view(nz, ny, nx).permute(2, 1, 0), b.view(nz, nx, ny).permute(1, 2, 0), rims


def _scatter(entry, lors, values, shape, center, size, tof, nsigma):
    """One call of a C entry on padded accumulators: the folded image."""
    from srf_gb300._lib import call, f32, f32x3, i32, i32x3, i64, i64x3, ptr, stream_ptr
    from srf_gb300.kernels import _tof_ptr
    bp, bt, rims = _padded(shape)
    head = [ptr(lors), i64(lors.shape[0]), i32(7)]
    tail = [ptr(values), ptr(bp), i64x3(bp.stride()), ptr(bt), i64x3(bt.stride()), i32x3(shape), f32x3(center), f32x3(size),
            stream_ptr(lors.device)]
    t = [_tof_ptr(lors) if tof else None, i32(7), f32(tof[0] if tof else 0.0), f32(tof[1] if tof else 0.0), f32(nsigma)]
    if entry == "adjoint":
        call("srf_projection_adjoint", *head, *t, *tail)
    elif tof:
        call("srf_backprojection_tof", *head, *t, *tail)
    else:
        call("srf_backprojection", *head, *tail)
    for r in rims:
        assert not r.any() and bool(torch.isfinite(r).all())
    return bp + bt


@pytest.mark.parametrize("shape,vox", [([64, 64, 16], (2.0, 2.0, 2.0)), ([41, 37, 9], (3.1, 2.7, 3.5)), ([150, 64, 7], (1.0, 2.0, 4.0))])
@pytest.mark.parametrize("tof,nsigma", [(None, 0.0), (TOF, 0.0), (TOF, 1.0)])
@pytest.mark.parametrize("entry", ["back", "adjoint"])
def test_scattered_values(cuda_lib, entry, tof, nsigma, shape, vox):
    center, size = [1.0, -2.0, 0.5], [a * b for a, b in zip(shape, vox)]
    lors = _lors(3001, 5)
    good = torch.rand(3001, device="cuda") + 0.5
    bad_rows = torch.arange(0, 3001, 5, device="cuda")  # all of the LORs beside the image ...
    bad_rows = torch.cat([bad_rows, torch.arange(1, 3001, 211, device="cuda")])  # ... and a few others
    values = good.clone()
    values[bad_rows] = torch.tensor(BAD, device="cuda").repeat(len(bad_rows) // 3 + 1)[:len(bad_rows)]
    only = torch.zeros_like(good)
    only[bad_rows] = 1.0
    rest = good.clone()
    rest[bad_rows] = 0.0
    args = (shape, center, size, tof, nsigma)
    got, touched, want = (_scatter(entry, lors, v, *args) for v in (values, only, rest))
    inside = touched != 0
    assert inside.any() and not inside.all()
    assert not torch.isfinite(got[inside]).any()
    assert bool(torch.isfinite(got[~inside]).all())
    assert rel_l2(got[~inside].cpu().numpy(), want[~inside].cpu().numpy()) <= TOL
    # LORs that visit nothing leave the image as it is
    beside = values.clone()
    beside[torch.arange(1, 3001, 211, device="cuda")] = 0.0
    beside[::5] = values[::5]
    one_beside = torch.zeros_like(good)
    one_beside[::5] = 1.0
    assert not _scatter(entry, lors, one_beside, *args).any()
    clean = torch.where(torch.isfinite(beside), beside, torch.zeros_like(good))
    got, want = _scatter(entry, lors, beside, *args), _scatter(entry, lors, clean, *args)
    assert bool(torch.isfinite(got).all()) and rel_l2(got.cpu().numpy(), want.cpu().numpy()) <= TOL


@pytest.mark.parametrize("shape,nsigma,tof,many", [([64, 64, 16], 3.0, TOF, False), ([64, 64, 16], 0.0, TOF, False),
                                                   ([101, 110, 9], 2.0, TOF, False), ([64, 60, 16], 0.0, None, False),
                                                   ([64, 64, 16], 3.0, TOF, True), ([64, 64, 16], 0.0, TOF, True),
                                                   ([101, 110, 9], 2.0, TOF, True)])
def test_subset_step_values(cuda_lib, shape, nsigma, tof, many):
    """The fused step (its chunk, rolled and two-walk forms) and the several-study kernel."""
    import ctypes
    from srf_gb300._lib import SRF_RATIO_PLAIN, call, f32, f32x3, i32, i32x3, i64, ptr, stream_ptr
    from srf_gb300.kernels import _tof_ptr
    vox = 128.0 / shape[0]
    center, size = [0.0, 0.0, 0.0], [128.0, shape[1] * vox, shape[2] * 2.0]
    lors = _lors(2003, 9)
    good = torch.rand(2003, device="cuda") + 0.5
    rows = torch.cat([torch.arange(0, 2003, 5), torch.arange(2, 2003, 173)]).cuda()
    nx, ny, nz = shape
    x = torch.rand(nz, ny, nx, device="cuda") + 0.5
    xt = x.permute(0, 2, 1).contiguous()

    def step(y):
        bp, bt, rims = _padded(shape)
        s = stream_ptr(lors.device)
        t = tof or (0.0, 0.0)
        if not many:
            call("srf_osem_subset", ptr(lors), i64(2003), i32(7), _tof_ptr(lors) if tof else None, i32(7), f32(t[0]), f32(t[1]),
                 f32(nsigma), ptr(y), None, i32(SRF_RATIO_PLAIN), f32(1e-3), ptr(x), ptr(xt), ptr(bp), ptr(bt), i32x3(shape),
                 f32x3(center), f32x3(size), None, s)
        else:
            from srf_gb300.studies import SrfStudy
            d = SrfStudy()
            d.lors, d.tof, d.y = lors.data_ptr(), lors.data_ptr() + 24, y.data_ptr()
            d.n, d.lor_stride, d.tof_stride = 2003, 7, 7
            d.x, d.x_t, d.bp, d.bp_t = x.data_ptr(), xt.data_ptr(), bp.data_ptr(), bt.data_ptr()
            d.emap = x.data_ptr()
            for a in range(3):
                d.grid[a], d.center[a], d.size[a] = shape[a], center[a], size[a]
            desc = torch.frombuffer(bytearray(ctypes.string_at(ctypes.byref(d), ctypes.sizeof(d))), dtype=torch.uint8).cuda()
            off = torch.tensor([0, 63, 0, 0], dtype=torch.int64, device="cuda")
            call("srf_osem_subset_batch", ptr(desc), i32(1), ptr(off), i64(63), i32(1), f32(t[0]), f32(t[1]), f32(nsigma),
                 i32(SRF_RATIO_PLAIN), f32(1e-3), None, s)
        for r in rims:
            assert not r.any() and bool(torch.isfinite(r).all())
        return bp + bt

    y, only, rest = good.clone(), torch.zeros_like(good), good.clone()
    y[rows] = torch.tensor(BAD, device="cuda").repeat(len(rows) // 3 + 1)[:len(rows)]
    only[rows] = 1.0
    rest[rows] = 0.0
    got, touched, want = step(y), step(only), step(rest)
    inside = touched != 0
    assert inside.any() and not inside.all()
    assert not torch.isfinite(got[inside]).any()
    assert bool(torch.isfinite(got[~inside]).all())
    assert rel_l2(got[~inside].cpu().numpy(), want[~inside].cpu().numpy()) <= TOL
