"""The two forms of the snap and of the crystal-pair histogram: from per-scanner tables with an FP32 index, and
the direct one (for scanners whose tables do not fit, and for every hit that the FP32 index does not decide).
The C entry takes the number of rings apart from the axial length, and only the choice of the form depends
on it here: the same hits go through both and must agree bit for bit, in gaps, beyond the ends, far away,
not finite, and within the FP32 index's margin of a border between crystals."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
MANY = 6000  # rings: more table entries than fit


def _scanner(which):
    import srf_gb300 as nef
    from srf_gb300 import synth
    if which == "small":
        return synth.scanner_small()
    if which == "clinical":
        return synth.scanner_clinical()
    return nef.PetEcatScanner(120.0, 135.0, 3, 12, 5.0, nef.Block([15.0, 40.0, 21.0], [1, 10, 7]), nef.TofConfig())  # with gaps


def _args(sc, rings):
    from srf_gb300._lib import ctypes
    b = sc.blocks
    d = (ctypes.c_double * 8)(sc.average_radius, sc.angle_per_block, sc.axial_length, sc.gap, b.size[1], b.size[2],
                              b.unit_size[1], b.unit_size[2])
    return d, (ctypes.c_int64 * 4)(b.shape[1], b.shape[2], sc.nb_blocks_per_ring, rings)


def _snap(lors, sc, rings, cols):
    from srf_gb300._lib import call, i32, i64, ptr, stream_ptr
    out = torch.full((lors.shape[0], cols), -1.0, device="cuda") if cols else None
    ids = torch.full((lors.shape[0], 2), -1, dtype=torch.int64, device="cuda")
    call("srf_listmode_snap", ptr(lors), i64(lors.shape[0]), i32(lors.stride(0)), *_args(sc, rings), ptr(out), i32(cols or 6),
         ptr(ids), stream_ptr(lors.device))
    return out, ids


def _hits(sc, n, seed):
    """(n, 3) hits: on crystals, on their borders to the last few ulps, in gaps, beyond the ends, anywhere."""
    rng = np.random.default_rng(seed)
    b, apb = sc.blocks, sc.angle_per_block
    blk = rng.integers(0, sc.nb_blocks_per_ring, n)
    ring = rng.integers(0, sc.nb_rings, n)
    iy, iz = rng.uniform(0, b.shape[1], n), rng.uniform(0, b.shape[2], n)
    kind = rng.integers(0, 8, n)
    eps = rng.choice([0.0, 1e-7, -1e-7, 1e-6, -1e-6, 1e-5, -1e-5], n)
    iy = np.where(kind == 1, np.round(iy) + eps, iy)
    iz = np.where(kind == 2, np.round(iz) + eps, iz)
    y = iy * b.unit_size[1] - b.size[1] / 2
    r = sc.average_radius + rng.uniform(-0.4, 0.4, n) * (sc.outer_radius - sc.inner_radius)
    th = blk * apb
    x = np.stack([r * np.cos(th) - y * np.sin(th), r * np.sin(th) + y * np.cos(th),
                  iz * b.unit_size[2] + ring * (sc.gap + b.size[2]) - sc.axial_length / 2], 1)
    x[kind == 3, 2] = rng.uniform(-1, 1, (kind == 3).sum()) * sc.axial_length          # half of them beyond the ends
    gap = kind == 4
    x[gap, 2] = ((ring[gap] + 1) * (sc.gap + b.size[2]) - rng.random(gap.sum()) * (sc.gap + 0.1) - sc.axial_length / 2)
    x[kind == 5] = rng.uniform(-1.5, 1.5, ((kind == 5).sum(), 3)) * sc.outer_radius       # anywhere, block corners among them
    x = x.astype(np.float32)
    near = kind == 6                                                                       # a few ulps about a border
    for _ in range(4):
        x[near, 2] = np.nextafter(x[near, 2], np.float32(rng.choice([-1e9, 1e9])))
    odd = np.flatnonzero(kind == 7)[:40]
    x[odd, rng.integers(0, 3, len(odd))] = rng.choice([np.nan, np.inf, -np.inf, 1e30, 0.0], len(odd)).astype(np.float32)
    return x


@pytest.mark.parametrize("which", ["small", "clinical", "gaps"])
@pytest.mark.parametrize("n", [31, 20011])
def test_snap_forms_agree(cuda_lib, which, n):
    sc = _scanner(which)
    lors = np.concatenate([_hits(sc, n, 1), _hits(sc, n, 2), np.arange(n, dtype=np.float32)[:, None]], 1).astype(np.float32)
    dev = torch.as_tensor(lors).cuda()
    for cols in (7, 6, 0):  # packed rows, plain rows, ids alone
        out, ids = _snap(dev, sc, sc.nb_rings, cols)
        want, want_ids = _snap(dev, sc, MANY, cols)
        assert torch.equal(ids, want_ids)
        if cols:
            assert torch.equal(out.view(torch.int32), want.view(torch.int32))


@pytest.mark.parametrize("which", ["small", "gaps"])
def test_histogram_forms_agree(cuda_lib, which):
    from srf_gb300._lib import call, i32, i64, ptr, stream_ptr
    sc = _scanner(which)
    lors = torch.as_tensor(np.concatenate([_hits(sc, 30011, 3), _hits(sc, 30011, 4)], 1)).cuda()
    bins = sc.nb_crystals * (sc.nb_crystals - 1) // 2
    got = []
    for rings in (sc.nb_rings, MANY):
        sino = torch.zeros(bins, dtype=torch.float64, device="cuda")
        dropped = torch.zeros(1, dtype=torch.int64, device="cuda")
        call("srf_lm2sino", ptr(lors), i64(lors.shape[0]), i32(6), None, *_args(sc, rings), ptr(sino), i64(bins), ptr(dropped),
             stream_ptr(lors.device))
        got.append((sino, int(dropped)))
    assert got[0][1] == got[1][1] > 0 and torch.equal(got[0][0], got[1][0])
    assert int(got[0][0].sum()) + got[0][1] == 30011


def test_scanner_beyond_the_tables(cuda_lib):
    import srf_gb300 as nef
    from srf_gb300 import kernels
    sc = nef.PetEcatScanner(400.0, 420.0, 2, 64, 0.0, nef.Block([20.0, 38.0, 16.0], [1, 40, 8]), nef.TofConfig())
    rng = np.random.default_rng(5)
    want = rng.integers(0, sc.nb_crystals, (5000, 2))
    pos = nef.EcatIndexToCrystalPos(sc)(np.arange(sc.nb_crystals))
    jit = rng.uniform(-0.3, 0.3, (5000, 6)) * min(sc.blocks.unit_size[1:])
    lors = torch.as_tensor((np.hstack([pos[want[:, 0]], pos[want[:, 1]]]) + jit).astype(np.float32)).cuda()
    out, ids = kernels.snap(lors, sc, want_ids=True)
    assert np.array_equal(ids.cpu().numpy(), want)
    assert np.abs(out.cpu().numpy() - np.hstack([pos[want[:, 0]], pos[want[:, 1]]])).max() <= 1e-4
