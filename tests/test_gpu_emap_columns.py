"""The sensitivity image from axial columns of the crystal table (srf_emap_block_full_ws) against the
oracle's line-by-line sum, at the sizes where the column kernel can go wrong: tiles of 32 slabs with
remainders, columns longer than the 64 members held at a time or than the axial window, an image
shorter than the scanner or off its centre, steep lines and slabs beyond the columns (straight into
the image), non-square voxels, single columns of unequal length, repeated
and non-finite rows, and tables without columns (line by line).

Tolerance 1e-5 relative L2, as for the line-by-line kernel: a line is traversed from one of its ends
instead of both, which moves face coordinates by their FP32 rounding (1.5e-5 voxel at 128), and a
voxel sums hundreds of lines."""
import numpy as np
import pytest
import torch

from conftest import rel_l2

pytestmark = pytest.mark.gpu
TOL = 1e-5


def _table(columns, members, radius, dz, seed):
    """(rows, 3): `columns` positions on a ring, each with members[k] crystals along z, in a shuffled order."""
    rng = np.random.default_rng(seed)
    rows = []
    for k in range(columns):
        a = 2 * np.pi * (k + 0.3) / columns
        n = members[k % len(members)]
        z = (np.arange(n) - (n - 1) / 2) * dz
        rows.append(np.stack([np.full(n, radius * np.cos(a)), np.full(n, radius * np.sin(a)), z], 1))
    t = np.concatenate(rows).astype(np.float32)
    return t[rng.permutation(len(t))]


CASES = [
    # shape, voxel sizes, centre, columns, members per column, axial pitch
    ([64, 64, 16], (2.0, 2.0, 2.0), (0, 0, 0), 40, [8], 4.0),
    ([33, 40, 7], (3.0, 3.0, 5.0), (0, 0, 0), 30, [9], 3.5),
    ([65, 31, 9], (1.9, 2.2, 2.0), (1.0, -2.0, 3.0), 24, [12], 4.0),      # z beyond both ends, non-square
    ([40, 40, 24], (3.0, 3.0, 1.5), (0, 0, 1.0), 10, [70, 65, 3], 0.6),    # longer than one piece, uneven
    ([40, 36, 5], (3.0, 3.0, 2.0), (0, 0, 0), 60, [5, 4], 40.0),          # steep lines, most of them outside
    ([40, 40, 130], (3.0, 3.0, 1.0), (0, 0, 0), 16, [31], 3.9),            # three pieces per column
    ([90, 90, 12], (3.0, 3.0, 3.0), (20.0, 0, 0), 20, [8], 4.0),          # the image reaches beyond the columns
    ([48, 48, 8], (2.5, 2.5, 3.0), (0, 0, 0), 120, [2], 5.0),             # short columns: line by line
]


@pytest.mark.parametrize("case", range(len(CASES)))
@pytest.mark.parametrize("use_t", [True, False])
def test_columns_match_oracle(cuda_lib, oracle, case, use_t):
    from srf_gb300 import _lib, kernels
    shape, vox, center, columns, members, dz = CASES[case]
    size = [n * v for n, v in zip(shape, vox)]
    table = _table(columns, members, 110.0, dz, case)
    if case == 0:  # a repeated row and a row that is not finite
        table = np.concatenate([table, table[:1], [[np.nan, 0, 0]], [[1, 2, np.inf]]]).astype(np.float32)
    finite = table[np.isfinite(table).all(1)]
    ref = oracle.emap_block_full(finite, 1, shape, list(center), size)
    dev = torch.as_tensor(table, device="cuda")
    if use_t:
        got = kernels.emap_block_full(dev, 1, shape, list(center), size)
    else:  # one view for both dominant axes
        got = kernels.new_xfast(shape, dev.device)
        need = _lib.load().srf_emap_workspace(_lib.i32(1), _lib.i32(len(table)))
        ws = torch.empty(need, dtype=torch.uint8, device="cuda")
        _lib.call("srf_emap_block_full_ws", _lib.ptr(dev), _lib.i32(1), _lib.i32(len(table)), _lib.ptr(got),
                  _lib.i64x3(got.stride()), None, None, _lib.i32x3(shape), _lib.f32x3(center), _lib.f32x3(size),
                  _lib.ptr(ws), _lib.i64(need), _lib.stream_ptr(dev.device))
    assert rel_l2(got.cpu().numpy(), ref) <= TOL


def test_workspace_is_checked(cuda_lib):
    from srf_gb300 import _lib
    shape = [16, 16, 4]
    dev = torch.zeros((32, 3), device="cuda")
    acc = torch.zeros(shape, device="cuda")
    need = _lib.load().srf_emap_workspace(_lib.i32(4), _lib.i32(8))
    assert need > 0
    args = lambda ws, n: (_lib.ptr(dev), _lib.i32(4), _lib.i32(8), _lib.ptr(acc), _lib.i64x3((64, 4, 1)), None, None,
                          _lib.i32x3(shape), _lib.f32x3((0, 0, 0)), _lib.f32x3((32, 32, 8)), ws, _lib.i64(n),
                          _lib.stream_ptr(dev.device))
    with pytest.raises(_lib.SrfError):
        _lib.call("srf_emap_block_full_ws", *args(None, need))
    with pytest.raises(_lib.SrfError):
        _lib.call("srf_emap_block_full_ws", *args(_lib.ptr(torch.empty(need, dtype=torch.uint8, device="cuda")), need - 1))
    assert _lib.load().srf_emap_workspace(_lib.i32(1 << 11), _lib.i32(1 << 10)) == 0  # line by line
