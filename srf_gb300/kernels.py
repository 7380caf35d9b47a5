"""Tensor-level entry points over the C ABI (device tensors in, device tensors out).

Layouts: images are handled as (nx, ny, nz) tensors of any strides. For speed the projector is
given an x-fastest view (memory order z, y, x; strides (1, nx, nx*ny)) for x-dominant LORs and a
y-fastest copy (memory order z, x, y) for y-dominant ones, so that the lanes of a LOR group touch
consecutive addresses; backprojections accumulate into the same two layouts and are folded once.
LORs are (N, >= 6) float32 rows with unit column stride; TOF values come from column 6.
"""
from __future__ import annotations

from typing import Optional, Sequence, Tuple

import torch

from . import _lib
from ._lib import call, f32, f32x3, i32, i32x3, i64, i64x3, ptr, stream_ptr

F32 = torch.float32


def _require_cuda(t: torch.Tensor, name: str) -> None:
    if not t.is_cuda:
        raise ValueError(f"{name} must be a CUDA tensor (srf_gb300 has no CPU path)")
    if t.dtype != F32:
        raise ValueError(f"{name} must be float32")


def check_lors(lors: torch.Tensor, tof: bool) -> Tuple[int, int]:
    _require_cuda(lors, "lors")
    if lors.dim() != 2 or lors.shape[1] < (7 if tof else 6):
        raise ValueError(f"lors must be (N, {'>=7' if tof else '>=6'}), got {tuple(lors.shape)}")
    if lors.stride(1) != 1 or lors.stride(0) < lors.shape[1]:
        raise ValueError("lors rows must be contiguous")
    return lors.shape[0], lors.stride(0)


def _tof_ptr(lors: torch.Tensor):
    return _lib.ctypes.c_void_p(lors.data_ptr() + 6 * 4)


def xfast(img: torch.Tensor) -> torch.Tensor:
    """(nx, ny, nz) view whose memory is x-fastest (a copy unless it already is)."""
    return img.permute(2, 1, 0).contiguous().permute(2, 1, 0)


def yfast(img: torch.Tensor) -> torch.Tensor:
    """(nx, ny, nz) view whose memory is y-fastest."""
    return img.permute(2, 0, 1).contiguous().permute(1, 2, 0)


def new_xfast(shape: Sequence[int], device) -> torch.Tensor:
    nx, ny, nz = shape
    return torch.zeros((nz, ny, nx), dtype=F32, device=device).permute(2, 1, 0)


def _relayout(shape, src: torch.Tensor, src2: Optional[torch.Tensor], dst: torch.Tensor,
              dst2: Optional[torch.Tensor] = None) -> None:
    """dst = src (+ src2), and dst2 the same: (nx, ny, nz) views of any strides, one pass."""
    st = lambda t: None if t is None else i64x3(t.stride())
    call("srf_relayout", ptr(src), st(src), ptr(src2), st(src2), ptr(dst), st(dst), ptr(dst2), st(dst2), i32x3(shape),
         stream_ptr(src.device))


def _empty_layout(shape, order: str, device) -> torch.Tensor:
    """Uninitialised (nx, ny, nz) view whose memory is x-, y- or z-fastest."""
    nx, ny, nz = shape
    if order == "x":
        return torch.empty((nz, ny, nx), dtype=F32, device=device).permute(2, 1, 0)
    if order == "y":
        return torch.empty((nz, nx, ny), dtype=F32, device=device).permute(1, 2, 0)
    return torch.empty((nx, ny, nz), dtype=F32, device=device)


def _projector_layouts(image: torch.Tensor, want_t: bool):
    """The x-fastest image (the image itself when it is) and, when wanted, its y-fastest copy."""
    shape = list(image.shape)
    have_x = image.stride(0) == 1
    if sum((n - 1) * s for n, s in zip(shape, image.stride())) >= 1 << 31:  # a view far beyond its own voxels
        image = image if have_x else xfast(image)
        return image, yfast(image) if want_t else None
    x = image if have_x else _empty_layout(shape, "x", image.device)
    t = _empty_layout(shape, "y", image.device) if want_t else None
    if not have_x:
        _relayout(shape, image, None, x, t)
    elif want_t:
        _relayout(shape, image, None, t)
    return x, t


def _accumulators(shape, device):
    """Zeroed x-fastest and y-fastest accumulators of one image."""
    nx, ny, nz = shape
    acc = torch.zeros((2, nz, ny * nx), dtype=F32, device=device)
    return acc[0].view(nz, ny, nx).permute(2, 1, 0), acc[1].view(nz, nx, ny).permute(1, 2, 0)


def _tof_args(tof_bin, tof_sigma2, nsigma):
    return f32(tof_bin), f32(tof_sigma2), f32(nsigma)


def project(lors: torch.Tensor, image: torch.Tensor, center, size, *, tof: Optional[Tuple[float, float]] = None,
            tof_nsigma: float = 0.0, image_t: Optional[torch.Tensor] = None,
            out: Optional[torch.Tensor] = None, make_t: bool = True) -> torch.Tensor:
    """p = A image for every LOR; tof = (tof_bin, tof_sigma2) selects the TOF projector."""
    n, stride = check_lors(lors, tof is not None)
    _require_cuda(image, "image")
    shape = list(image.shape)
    if image.dim() != 3:
        raise ValueError("image must be (nx, ny, nz)")
    image, made_t = _projector_layouts(image, image_t is None and make_t)
    image_t = made_t if image_t is None else image_t
    if out is None:
        out = torch.empty(n, dtype=F32, device=lors.device)
    st = i64x3(image.stride())
    t_args = (ptr(image_t), i64x3(image_t.stride())) if image_t is not None else (None, None)
    s = stream_ptr(lors.device)
    if tof is None:
        call("srf_projection", ptr(lors), i64(n), i32(stride), ptr(image), st, *t_args,
             i32x3(shape), f32x3(center), f32x3(size), ptr(out), s)
    else:
        call("srf_projection_tof", ptr(lors), i64(n), i32(stride), _tof_ptr(lors), i32(stride),
             *_tof_args(tof[0], tof[1], tof_nsigma), ptr(image), st, *t_args,
             i32x3(shape), f32x3(center), f32x3(size), ptr(out), s)
    return out


def backproject(lors: torch.Tensor, values: torch.Tensor, shape, center, size, *,
                tof: Optional[Tuple[float, float]] = None, tof_nsigma: float = 0.0,
                adjoint: bool = False, use_t: bool = True, order: str = "x") -> torch.Tensor:
    """A_bp^T values as an x-fastest (nx, ny, nz) tensor (order 'z': a contiguous one; adjoint=True:
    exact adjoint of ``project``)."""
    n, stride = check_lors(lors, tof is not None)
    _require_cuda(values, "values")
    values = values.contiguous()
    if values.numel() != n:
        raise ValueError("values must have one entry per LOR")
    shape = list(shape)
    acc, acc_t = _accumulators(shape, lors.device) if use_t else (new_xfast(shape, lors.device), None)
    st = i64x3(acc.stride())
    t_args = (ptr(acc_t), i64x3(acc_t.stride())) if acc_t is not None else (None, None)
    s = stream_ptr(lors.device)
    if adjoint:
        tof_p = _tof_ptr(lors) if tof is not None else None
        tb, ts = tof if tof is not None else (0.0, 0.0)
        call("srf_projection_adjoint", ptr(lors), i64(n), i32(stride), tof_p, i32(stride),
             *_tof_args(tb, ts, tof_nsigma), ptr(values), ptr(acc), st, *t_args,
             i32x3(shape), f32x3(center), f32x3(size), s)
    elif tof is None:
        call("srf_backprojection", ptr(lors), i64(n), i32(stride), ptr(values), ptr(acc), st,
             *t_args, i32x3(shape), f32x3(center), f32x3(size), s)
    else:
        call("srf_backprojection_tof", ptr(lors), i64(n), i32(stride), _tof_ptr(lors), i32(stride),
             *_tof_args(tof[0], tof[1], tof_nsigma), ptr(values), ptr(acc), st, *t_args,
             i32x3(shape), f32x3(center), f32x3(size), s)
    return _folded(shape, acc, acc_t, order)


def _folded(shape, acc: torch.Tensor, acc_t: Optional[torch.Tensor], order: str) -> torch.Tensor:
    """The two accumulators as one image."""
    if acc_t is None and order == "x":
        return acc
    out = _empty_layout(shape, order, acc.device)
    _relayout(shape, acc, acc_t, out)
    return out


MAX_BATCH = 8


def _width(B: int, shape) -> int:
    """Values per voxel of the interleaved layout for B images; 0: the separate-image kernels (one image,
    or so many voxels that element offsets would leave 31 bits)."""
    w = 0 if B < 2 else 2 if B == 2 else 4 if B <= 4 else 8
    return w if w * shape[0] * shape[1] * shape[2] < 1 << 31 else 0


def _interleaved(shape, width: int, device, fill: bool):
    """Interleaved buffers: x-fastest, and y-fastest for the y-dominant LORs. Images to read need the second one
    only where a voxel is less than a 32-byte sector; accumulators (fill) always have both: one sum over
    both kinds of LORs would round twice as much (rms) as the two."""
    nx, ny, nz = shape
    new = torch.zeros if fill else torch.empty
    il = new((nz, ny, nx, width), dtype=F32, device=device)
    return il, (new((nz, nx, ny, width), dtype=F32, device=device) if fill or width < 8 else None)


def project_batch(lors: torch.Tensor, images: torch.Tensor, center, size, *,
                  tof: Optional[Tuple[float, float]] = None, tof_nsigma: float = 0.0) -> torch.Tensor:
    """(B, N) projections of a batch of (nx, ny, nz) images (B <= 8), one traversal per LOR."""
    n, stride = check_lors(lors, tof is not None)
    _require_cuda(images, "images")
    if images.dim() != 4 or not 1 <= images.shape[0] <= MAX_BATCH:
        raise ValueError(f"images must be (B <= {MAX_BATCH}, nx, ny, nz)")
    B, nx, ny, nz = images.shape
    out = torch.empty((B, n), dtype=F32, device=lors.device)
    if B == 1:
        project(lors, images[0], center, size, tof=tof, tof_nsigma=tof_nsigma, out=out[0])
        return out
    s = stream_ptr(lors.device)
    tof_p = _tof_ptr(lors) if tof is not None else None
    tb, tsg = tof if tof is not None else (0.0, 0.0)
    w = _width(B, (nx, ny, nz))
    if w:
        il, il_t = _interleaved((nx, ny, nz), w, lors.device, fill=False)
        call("srf_interleave", ptr(images), i64(images.stride(0)), i64x3(images.stride()[1:]), i32(B), i32(w),
             i32x3((nx, ny, nz)), ptr(il), ptr(il_t), s)
        call("srf_projection_il", ptr(lors), i64(n), i32(stride), tof_p, i32(stride), *_tof_args(tb, tsg, tof_nsigma),
             i32(B), i32(w), ptr(il), ptr(il_t), i32x3((nx, ny, nz)), f32x3(center), f32x3(size), ptr(out), i64(n), s)
        return out
    xb = images.permute(0, 3, 2, 1).contiguous()             # (B, nz, ny, nx): x fastest
    yb = images.permute(0, 3, 1, 2).contiguous()             # (B, nz, nx, ny): y fastest
    call("srf_projection_batch", ptr(lors), i64(n), i32(stride), tof_p, i32(stride),
         *_tof_args(tb, tsg, tof_nsigma), i32(B), i64(nx * ny * nz), ptr(xb), i64x3((1, nx, nx * ny)),
         ptr(yb), i64x3((ny, 1, nx * ny)), i32x3((nx, ny, nz)), f32x3(center), f32x3(size), ptr(out),
         i64(n), s)
    return out


def adjoint_batch(lors: torch.Tensor, values: torch.Tensor, shape, center, size, *,
                  tof: Optional[Tuple[float, float]] = None, tof_nsigma: float = 0.0) -> torch.Tensor:
    """(B, nx, ny, nz) exact adjoint of ``project_batch`` for (B, N) LOR values."""
    n, stride = check_lors(lors, tof is not None)
    _require_cuda(values, "values")
    values = values.contiguous()
    if values.dim() != 2 or values.shape[1] != n or not 1 <= values.shape[0] <= MAX_BATCH:
        raise ValueError(f"values must be (B <= {MAX_BATCH}, N)")
    B = values.shape[0]
    nx, ny, nz = shape
    if B == 1:
        return backproject(lors, values[0], shape, center, size, tof=tof, tof_nsigma=tof_nsigma, adjoint=True)[None]
    s = stream_ptr(lors.device)
    tof_p = _tof_ptr(lors) if tof is not None else None
    tb, tsg = tof if tof is not None else (0.0, 0.0)
    w = _width(B, shape)
    if w:
        il, il_t = _interleaved(shape, w, lors.device, fill=True)
        call("srf_projection_adjoint_il", ptr(lors), i64(n), i32(stride), tof_p, i32(stride),
             *_tof_args(tb, tsg, tof_nsigma), i32(B), i32(w), ptr(values), i64(n), ptr(il), ptr(il_t), i32x3(shape),
             f32x3(center), f32x3(size), s)
        out = torch.empty((B, nx, ny, nz), dtype=F32, device=lors.device)
        call("srf_deinterleave", ptr(il), ptr(il_t), i32(B), i32(w), i32x3(shape), ptr(out), i64(out.stride(0)),
             i64x3(out.stride()[1:]), s)
        return out
    acc = torch.zeros((B, nz, ny, nx), dtype=F32, device=lors.device)
    acc_t = torch.zeros((B, nz, nx, ny), dtype=F32, device=lors.device)
    call("srf_projection_adjoint_batch", ptr(lors), i64(n), i32(stride), tof_p, i32(stride),
         *_tof_args(tb, tsg, tof_nsigma), i32(B), ptr(values), i64(n), ptr(acc), i64(nx * ny * nz),
         i64x3((1, nx, nx * ny)), ptr(acc_t), i64x3((ny, 1, nx * ny)), i32x3(shape), f32x3(center),
         f32x3(size), s)
    out = acc.permute(0, 3, 2, 1)                             # (B, nx, ny, nz) views, x fastest
    for b in range(B):
        fold(out[b], acc_t[b].permute(1, 2, 0))
    return out


def count_pairs(lors: torch.Tensor, shape, center, size, *, rules: int,
                tof: Optional[Tuple[float, float]] = None, tof_nsigma: float = 0.0) -> int:
    """Exact number of (LOR, voxel) visits of the projector (rules=0) or backprojector (1)."""
    n, stride = check_lors(lors, tof is not None)
    cnt = torch.zeros(1, dtype=torch.int64, device=lors.device)
    tof_p = _tof_ptr(lors) if tof is not None else None
    tb, ts = tof if tof is not None else (0.0, 0.0)
    call("srf_count_pairs", ptr(lors), i64(n), i32(stride), tof_p, i32(stride),
         *_tof_args(tb, ts, tof_nsigma), i32(rules), i32x3(shape), f32x3(center), f32x3(size),
         ptr(cnt), stream_ptr(lors.device))
    return int(cnt.item())


def fold(dst: torch.Tensor, src: torch.Tensor) -> None:
    call("srf_fold_views", ptr(dst), i64x3(dst.stride()), ptr(src), i64x3(src.stride()),
         i32x3(dst.shape), stream_ptr(dst.device))


def copy_view(dst: torch.Tensor, src: torch.Tensor) -> None:
    call("srf_copy_view", ptr(dst), i64x3(dst.stride()), ptr(src), i64x3(src.stride()),
         i32x3(dst.shape), stream_ptr(dst.device))


class SubsetState:
    """Device state of a list-mode MLEM/OSEM reconstruction: x (x-fastest) and its y-fastest copy,
    two backprojection accumulators and an FP64 log-likelihood accumulator."""

    def __init__(self, shape, center, size, device, x0: Optional[torch.Tensor] = None):
        self.shape, self.center, self.size = list(shape), list(center), list(size)
        nx, ny, nz = self.shape
        if x0 is None:
            one = torch.ones((2, nz, ny * nx), dtype=F32, device=device)
            self.x = one[0].view(nz, ny, nx).permute(2, 1, 0)
            self.x_t = one[1].view(nz, nx, ny).permute(1, 2, 0)
        else:
            self.x = new_xfast(shape, device)
            self.x.copy_(x0)
            self.x_t = yfast(self.x)
        # both backprojection accumulators in one flat buffer (one collective sums both)
        v = nx * ny * nz
        self._acc = torch.zeros(2 * v, dtype=F32, device=device)
        self.bp = self._acc[:v].view(nz, ny, nx).permute(2, 1, 0)
        self.bp_t = self._acc[v:].view(nz, nx, ny).permute(1, 2, 0)
        self.loglik = torch.zeros(1, dtype=torch.float64, device=device)

    def image(self) -> torch.Tensor:
        """A contiguous (nx, ny, nz) copy of x."""
        out = _empty_layout(self.shape, "z", self.x.device)
        _relayout(self.shape, self.x, None, out)
        return out

    def accumulators(self) -> torch.Tensor:
        """The flat buffer holding both backprojection accumulators (what an event-sharded
        reconstruction sums over its ranks before the update)."""
        return self._acc

    def subset(self, lors: torch.Tensor, y: Optional[torch.Tensor], *, rule: int, eps: float,
               tof: Optional[Tuple[float, float]] = None, tof_nsigma: float = 0.0,
               track_loglik: bool = False, add: Optional[torch.Tensor] = None) -> None:
        n, stride = check_lors(lors, tof is not None)
        if y is not None:
            _require_cuda(y, "y")
        tof_p = _tof_ptr(lors) if tof is not None else None
        tb, ts = tof if tof is not None else (0.0, 0.0)
        call("srf_osem_subset", ptr(lors), i64(n), i32(stride), tof_p, i32(stride),
             *_tof_args(tb, ts, tof_nsigma), ptr(y), ptr(add), i32(rule), f32(eps), ptr(self.x),
             ptr(self.x_t), ptr(self.bp), ptr(self.bp_t), i32x3(self.shape),
             f32x3(self.center), f32x3(self.size), ptr(self.loglik) if track_loglik else None,
             stream_ptr(lors.device))

    def update(self, emap_xfast: torch.Tensor, guard_zero: bool) -> None:
        call("srf_osem_update", ptr(self.x), ptr(self.x_t), ptr(self.bp), ptr(self.bp_t),
             ptr(emap_xfast), i32(1 if guard_zero else 0), i32x3(self.shape),
             stream_ptr(self.x.device))


def emap_block_full(table: torch.Tensor, n_blocks: int, shape, center, size, order: str = "x") -> torch.Tensor:
    _require_cuda(table, "crystal table")
    m = table.shape[0] // n_blocks
    shape = list(shape)
    acc, acc_t = _accumulators(shape, table.device)
    need = int(_lib.load().srf_emap_workspace(i32(n_blocks), i32(m)))
    ws = torch.empty(need, dtype=torch.uint8, device=table.device) if need else None
    call("srf_emap_block_full_ws", ptr(table), i32(n_blocks), i32(m), ptr(acc), i64x3(acc.stride()),
         ptr(acc_t), i64x3(acc_t.stride()), i32x3(shape), f32x3(center), f32x3(size), ptr(ws), i64(need),
         stream_ptr(table.device))
    return _folded(shape, acc, acc_t, order)


def sss(pairs: torch.Tensor, crystal_pos: torch.Tensor, scatter_pos: torch.Tensor,
        sumup_emission: torch.Tensor, atten: torch.Tensor, umap: torch.Tensor, umap_size,
        nb_crystals_per_ring: int, nb_blocks_per_ring: int, grid_block, low_energy: int,
        high_energy: int, resolution: float) -> Tuple[torch.Tensor, torch.Tensor]:
    dev = pairs.device
    n = pairs.shape[0]
    scatter = torch.empty(n, dtype=F32, device=dev)
    scale = torch.empty(n, dtype=F32, device=dev)
    umap = umap.contiguous()
    call("srf_sss", ptr(pairs.contiguous()), i64(n), ptr(crystal_pos.contiguous()),
         i32(crystal_pos.shape[0]), ptr(scatter_pos.contiguous()), i32(scatter_pos.shape[0]),
         ptr(sumup_emission.contiguous()), ptr(atten.contiguous()), ptr(umap),
         i32x3(umap.shape), f32x3(umap_size), i32(nb_crystals_per_ring), i32(nb_blocks_per_ring),
         i32x3(grid_block), i32(low_energy), i32(high_energy), f32(resolution), ptr(scatter),
         ptr(scale), stream_ptr(dev))
    return scatter, scale


# ---------------------------------------------------------------- list-mode ingestion

def scanner_args(scanner):
    """(double[8], int64[4]) description of a PetEcatScanner for the list-mode kernels."""
    import ctypes
    b = scanner.blocks
    d = (ctypes.c_double * 8)(scanner.average_radius, scanner.angle_per_block, scanner.axial_length,
                              scanner.gap, b.size[1], b.size[2], b.unit_size[1], b.unit_size[2])
    s = (ctypes.c_int64 * 4)(int(b.shape[1]), int(b.shape[2]), int(scanner.nb_blocks_per_ring),
                             int(scanner.nb_rings))
    return d, s


def snap(lors: torch.Tensor, scanner, want_ids: bool = False, out: Optional[torch.Tensor] = None):
    """Endpoints snapped to crystal centres (columns 6 .. out's width - 1 kept); optionally the
    crystal ids. ``out`` (N, >= 6) float32 rows with unit column stride, default like ``lors``."""
    _require_cuda(lors, "lors")
    n, stride = lors.shape[0], lors.stride(0)
    if lors.dim() != 2 or lors.shape[1] < 6 or lors.stride(1) != 1:
        raise ValueError("lors must be (N, >= 6) rows with unit column stride")
    if out is None:
        out = torch.empty_like(lors)
    else:
        _require_cuda(out, "out")
        if out.dim() != 2 or out.shape[0] != n or out.shape[1] < 6 or out.stride(1) != 1 \
                or out.stride(0) < out.shape[1] or out.device != lors.device:
            raise ValueError("out must be (N, >= 6) rows with unit column stride on the LORs' device")
    ids = torch.empty((n, 2), dtype=torch.int64, device=lors.device) if want_ids else None
    d, s = scanner_args(scanner)
    call("srf_listmode_snap", ptr(lors), i64(n), i32(stride), d, s, ptr(out), i32(out.stride(0)),
         ptr(ids), stream_ptr(lors.device))
    return (out, ids) if want_ids else out


def lm2sino(lors: torch.Tensor, values: Optional[torch.Tensor], scanner) -> Tuple[torch.Tensor, int]:
    """Triangular crystal-pair sinogram (float64, n(n-1)/2 bins) and the number of dropped events."""
    _require_cuda(lors, "lors")
    nc = scanner.nb_crystals
    sino = torch.zeros(nc * (nc - 1) // 2, dtype=torch.float64, device=lors.device)
    dropped = torch.zeros(1, dtype=torch.int64, device=lors.device)
    d, s = scanner_args(scanner)
    call("srf_lm2sino", ptr(lors), i64(lors.shape[0]), i32(lors.stride(0)),
         ptr(values.contiguous() if values is not None else None), d, s, ptr(sino), i64(sino.numel()),
         ptr(dropped), stream_ptr(lors.device))
    return sino, int(dropped.item())


def attenuation(lors: torch.Tensor, umap: torch.Tensor, center, size,
                values: Optional[torch.Tensor] = None) -> torch.Tensor:
    """exp(-(P mu) L^2 / unit) per LOR, or values / that (AttenuationCorrect) when values given."""
    n, stride = check_lors(lors, False)
    _require_cuda(umap, "umap")
    if umap.stride(0) != 1:
        umap = xfast(umap)
    out = torch.empty(n, dtype=F32, device=lors.device)
    call("srf_attenuation", ptr(lors), i64(n), i32(stride), ptr(umap), i64x3(umap.stride()),
         i32x3(umap.shape), f32x3(center), f32x3(size),
         ptr(values.contiguous() if values is not None else None), ptr(out), stream_ptr(lors.device))
    return out
