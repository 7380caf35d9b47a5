"""Performance cases of the list-mode reconstruction path, through the package's public classes.

A case is one call that a reconstruction program makes: a projection or a backprojection, an MLEM
job, one OSEM pass, a training step of the differentiable projector, a sensitivity image, a scatter
sinogram, the snapping of raw list mode, or the replay of a batch of studies. Scanners, phantoms and
sizes are those of the repository's own workloads (``srf_gb300.synth``, ``bench.py``): the
640-crystal scanner with its 64 x 64 x 16 image, the clinical scanner (32,448 crystals, 530 ps TOF)
with its 200 x 200 x 109 image, and odd sizes between them.

``listed()`` gives the fixed cases, ``draw(rng)`` one more of the same ranges, ``prepare`` the
resident inputs of a case, ``run`` one pass, ``work`` the bytes and operations that a pass cannot do
without, and ``exact`` the same results in 64 bits from plain torch.
"""
import math

import numpy as np
import torch

import srf_gb300 as nef
from srf_gb300 import autograd, scatter_sinogram, studies, synth

# ------------------------------------------------------------------ the cases


def listed():
    """The fixed cases, from the smallest call to the largest reconstruction pass."""
    return [
        # interactive use: a few thousand LORs of a preclinical scanner projected once, where the
        # launches and the image's layout copies are the whole cost
        dict(name="project_small", kind="project", scanner="small", nx=64, ny=64, nz=16, vox=2.0, aspect=1.0,
             events=3000, tof=False, nsigma=0.0),
        # the preclinical job: 10 MLEM iterations over 1e5 events
        dict(name="mlem_small", kind="mlem", scanner="small", nx=64, ny=64, nz=16, vox=2.0, aspect=1.0,
             events=100000, iters=10),
        # the headline: one OSEM pass at clinical size, 2e7 events kept in acquisition order
        dict(name="osem_tof_clinical", kind="osem", scanner="clinical", nx=200, ny=200, nz=109, vox=2.04, aspect=1.0,
             events=20000000, subsets=10, order="interleaved", nsigma=3.0, add=False),
        # a short acquisition on an odd grid with non-square voxels, permuted subsets and a scatter term
        dict(name="osem_tof_odd", kind="osem", scanner="clinical", nx=143, ny=161, nz=77, vox=2.7, aspect=1.1,
             events=700001, subsets=7, order="random", nsigma=3.0, add=True),
        # the TOF projector with its default, untruncated kernel
        dict(name="project_tof_clinical", kind="project", scanner="clinical", nx=200, ny=200, nz=109, vox=2.04,
             aspect=1.0, events=1000000, tof=True, nsigma=0.0),
        # the plain backprojector over long LORs
        dict(name="backproject_clinical", kind="backproject", scanner="clinical", nx=200, ny=200, nz=109, vox=2.04,
             aspect=1.0, events=2000000, tof=False, nsigma=0.0),
        # a training step of a learned method: 8 images, forward, Poisson loss, backward
        dict(name="autograd_batch8", kind="autograd", scanner="clinical", nx=128, ny=128, nz=64, vox=3.2, aspect=1.0,
             events=5000000, images=8, tof=True, nsigma=3.0),
        # a gradient of one image (a regularised reconstruction by gradient descent), non-TOF, odd grid
        dict(name="autograd_one_odd", kind="autograd", scanner="clinical", nx=97, ny=90, nz=47, vox=4.1, aspect=1.0,
             events=300007, images=1, tof=False, nsigma=0.0),
        # the sensitivity image of the clinical scanner, 1.05e9 crystal pairs, once per geometry
        dict(name="emap_clinical", kind="emap", radius=424.0, blocks=48, crystals=13, rings=4, crystal_mm=4.0,
             nx=200, ny=200, nz=109, vox=2.04),
        # single-scatter simulation of the whole coarse sinogram (bins = 0: all of them)
        dict(name="sss_coarse", kind="sss", bins=0),
        # raw list mode of one acquisition chunk snapped to crystal centres
        dict(name="snap_chunk", kind="snap", scanner="clinical", events=2000000),
        # several uneven studies of a worklist, two OSEM iterations of four subsets, as one graph
        dict(name="studies_uneven", kind="studies", studies=12, low=100000, high=2000000, subsets=4, iters=2, pick=1),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: sizes log-uniform over the listed ranges, most of them odd."""
    kind = rng.choice(["project", "project", "backproject", "osem", "osem", "mlem", "autograd", "autograd",
                       "emap", "sss", "snap", "studies"])
    if kind == "snap":
        return dict(kind=kind, scanner=rng.choice(["small", "clinical"]), events=_log(rng, 2000, 4000000))
    if kind == "sss":
        return dict(kind=kind, bins=_log(rng, 2048, 800000))
    if kind == "studies":
        return dict(kind=kind, studies=rng.randint(3, 12), low=100000, high=_log(rng, 200000, 2000000),
                    subsets=rng.randint(2, 6), iters=rng.randint(1, 2), pick=rng.randint(2, 1 << 20))
    if kind == "emap":
        small = rng.random() < 0.5
        vox = rng.uniform(1.6, 2.4) if small else rng.uniform(2.0, 5.0)
        n = rng.randint(40, 80) if small else rng.randint(80, 200)
        return dict(kind=kind, radius=99.0 if small else 424.0, blocks=16 if small else rng.choice([16, 24, 32, 48]),
                    crystals=4 if small else rng.randint(3, 9), rings=rng.randint(1, 4),
                    crystal_mm=3.2 if small else 4.0, nx=n, ny=n, nz=rng.randint(8, 24) if small else rng.randint(24, 109),
                    vox=round(vox, 3))
    clinical = kind == "osem" or rng.random() < 0.6
    c = dict(kind=kind, scanner="clinical" if clinical else "small")
    if clinical:
        fov = rng.uniform(300.0, 410.0)
        c["nx"] = _log(rng, 80, 200)
        c["nz"] = rng.randint(40, 109)
    else:
        fov = rng.uniform(100.0, 128.0)
        c["nx"] = _log(rng, 48, 96)
        c["nz"] = rng.randint(11, 24)
    c["aspect"] = rng.choice([1.0, 1.0, 1.0, round(rng.uniform(0.85, 1.15), 3)])  # dy / dx
    c["vox"] = round(fov / c["nx"], 3)
    c["ny"] = c["nx"] if rng.random() < 0.5 else max(40, int(c["nx"] * rng.uniform(0.8, 1.0)))
    if kind == "mlem":
        c.update(events=_log(rng, 20000, 400000), iters=rng.randint(4, 12))
    elif kind == "osem":
        c.update(events=_log(rng, 100000, 12000000), subsets=rng.randint(2, 12),
                 order=rng.choice(["interleaved", "random"]), nsigma=rng.choice([3.0, 3.0, 0.0]),
                 add=rng.random() < 0.4)
    else:
        c.update(tof=rng.random() < 0.6, nsigma=0.0)
        if c["tof"] and rng.random() < 0.5:
            c["nsigma"] = 3.0
        if kind == "autograd":
            c["images"] = rng.choice([1, 1, 2, 3, 4, 5, 6, 7, 8, 8])
            c["events"] = _log(rng, 20000, 2000000)
        else:
            c["events"] = _log(rng, 2000, 3000000)
    return c


# ------------------------------------------------------------------ inputs


def _dev():
    return torch.device("cuda", torch.cuda.current_device())


def _scanner(case):
    return synth.scanner_small() if case["scanner"] == "small" else synth.scanner_clinical()


def _image_config(case):
    vx, vy = case["vox"], case["vox"] * case.get("aspect", 1.0)
    vz = 2.0 if case.get("scanner") == "small" else 2.03 * case["vox"] / 2.04
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    return nef.ImageConfig([nx, ny, nz], [0.0, 0.0, 0.0], [nx * vx, ny * vy, nz * vz])


def _phantom(case, ic, seed):
    if case.get("scanner") == "small":
        return synth.phantom_cylinder(ic, device=_dev())
    return synth.phantom_body(ic, seed=seed, device=_dev(), max_lesions=16)


def _events(scanner, ic, act, n, seed):
    chunk = min(1 << 22, max(16384, 8 * n))
    return synth.sample_events(scanner, ic, act, n, seed=seed, tof_fwhm_ps=530.0, device=_dev(), chunk=chunk)


def _rand(seed, *shape):
    g = torch.Generator(device=_dev()).manual_seed(seed)
    return torch.rand(*shape, generator=g, device=_dev())


def _sensitivity(scanner, ic, n, mean_y, eff_len, seed):
    """A smooth sensitivity image (falling towards the axial ends and the edge of the field of view) at
    a level that puts the reconstructed image near 50."""
    nx, ny, nz = ic.shape
    dev = _dev()
    x = (torch.arange(nx, device=dev) + 0.5) / nx * 2 - 1
    y = (torch.arange(ny, device=dev) + 0.5) / ny * 2 - 1
    z = (torch.arange(nz, device=dev) + 0.5) / nz * 2 - 1
    g = _rand(seed, 3).tolist()
    r2 = x[:, None, None] ** 2 + y[None, :, None] ** 2
    prof = (1 - (0.25 + 0.1 * g[0]) * r2) * (1 - (0.5 + 0.2 * g[1]) * z.abs()[None, None, :])
    L = 2 * scanner.average_radius / ic.unit_size[0]
    level = n * mean_y * L * L / (nx * ny * nz * eff_len) / 50.0
    return (prof * (level * (0.9 + 0.2 * g[2]))).contiguous()


def _prep_events(case, seed):
    sc, ic = _scanner(case), _image_config(case)
    act = _phantom(case, ic, seed)
    return sc, ic, act, _events(sc, ic, act, case["events"], seed + 1)


def _study_list(case):
    """(shape, voxel mm, events) of each study, fixed by the case."""
    rng = np.random.default_rng(case["pick"])
    shapes = [(64, 64, 64), (96, 96, 64), (128, 128, 80), (160, 160, 80)]
    out = []
    for _ in range(case["studies"]):
        shape = shapes[int(rng.integers(0, 4))]
        vox = float(rng.choice([2.0, 3.0, 4.0]))
        n = int(round(math.exp(rng.uniform(math.log(case["low"]), math.log(case["high"])))))
        out.append((shape, vox, n))
    return out


def _study_inputs(case, seed):
    sc = synth.scanner_clinical()
    out = []
    for j, (shape, vox, n) in enumerate(_study_list(case)):
        ic = nef.ImageConfig(list(shape), [0.0, 0.0, 0.0], [s * vox for s in shape])
        act = synth.phantom_body(ic, seed=seed + j, device=_dev(), max_lesions=8)
        lors = _events(sc, ic, act, n, seed + 100 + j)
        em = _sensitivity(sc, ic, n, 1.0, sc.tof.tof_bin, seed + 200 + j) / case["subsets"]
        out.append((ic, lors, em))
    return sc, out


def _raw_hits(case, seed):
    """Unsnapped list mode: crystal hits spread over the crystal's face and depth."""
    sc = _scanner(case)
    ic = synth.image_small() if case["scanner"] == "small" else synth.image_clinical()
    lors = _events(sc, ic, _phantom(case, ic, seed), case["events"], seed + 1)
    n = lors.shape[0]
    u = (_rand(seed + 2, n, 2, 3) - 0.5) * 0.98
    apb = sc.angle_per_block
    out = lors.clone()
    for k in range(2):
        p = lors[:, 3 * k:3 * k + 3].double()
        ang = torch.round(torch.atan2(p[:, 1], p[:, 0]) / apb) * apb
        d = u[:, k, 0].double() * (sc.outer_radius - sc.inner_radius)
        t = u[:, k, 1].double() * sc.blocks.unit_size[1]
        out[:, 3 * k] = (p[:, 0] + d * torch.cos(ang) - t * torch.sin(ang)).float()
        out[:, 3 * k + 1] = (p[:, 1] + d * torch.sin(ang) + t * torch.cos(ang)).float()
        out[:, 3 * k + 2] = (p[:, 2] + u[:, k, 2].double() * sc.blocks.unit_size[2]).float()
    return sc, out


def _emap_scanner(case, seed):
    # the radius of the installed detector ring, a little different from one scanner to the next
    r = case["radius"] + 0.5 * float(np.random.default_rng(seed).random())
    w = case["crystals"] * case["crystal_mm"]
    return nef.PetEcatScanner(r, r + 20.0, case["rings"], case["blocks"], 0.0,
                              nef.Block([20.0, w, w], [1, case["crystals"], case["crystals"]]), nef.TofConfig())


def prepare(case, seed):
    """The resident inputs of a case, from the seed alone."""
    kind = case["kind"]
    s = dict(kind=kind, case=case)
    if kind == "snap":
        sc, raw = _raw_hits(case, seed)
        s.update(trans=nef.PetEcatListmodeTrans(sc), sc=sc, lors=raw,
                 lm=nef.Listmode(torch.ones(raw.shape[0], device=_dev()), nef.Lors(raw)))
    elif kind == "emap":
        sc = _emap_scanner(case, seed)
        ic = _image_config(case)
        s.update(sc=sc, ic=ic, gen=nef.EmapGenerator("block-full", sc),
                 image=nef.Image(torch.empty(ic.shape, device=_dev()), ic.center, ic.size))
    elif kind == "sss":
        geo = scatter_sinogram.CoarseGeometry(synth.scanner_clinical(), device=_dev())
        em, mu = scatter_sinogram.random_phantom(seed, device=_dev())
        bins = None
        if case["bins"]:
            bins = torch.randperm(geo.n_bins(), generator=torch.Generator(device=_dev()).manual_seed(seed),
                                  device=_dev())[:case["bins"]]
        s.update(geo=geo, em=em, mu=mu, bins=bins)
    elif kind == "studies":
        sc, inputs = _study_inputs(case, seed)
        tof = (sc.tof.tof_bin, sc.tof.tof_sigma2)
        todo = [studies.Study(lors, ic.shape, ic.center, ic.size, em.permute(2, 1, 0).contiguous().permute(2, 1, 0))
                for ic, lors, em in inputs]
        batch = studies.StudyBatch(todo, case["subsets"], tof, tof_nsigma=3.0)
        batch.capture(concurrent=True)
        s.update(batch=batch)
    else:
        sc, ic, act, lors = _prep_events(case, seed)
        n = lors.shape[0]
        tof = case.get("tof", kind == "osem")
        lors = lors if tof else lors[:, :6].contiguous()
        s.update(sc=sc, ic=ic, lors=lors)
        if kind in ("project", "backproject"):
            image = nef.Image((act + 0.1).contiguous(), ic.center, ic.size)
            fwd, back = nef.Project("tf"), nef.BackProject("tf")
            if tof:
                fwd = nef.ProjectTof("tf", sc.tof, case["nsigma"])
                back = nef.BackProjectTof("tf", sc.tof, case["nsigma"])
            s.update(image=image, op=fwd if kind == "project" else back,
                     lm=nef.Listmode(_rand(seed + 3, n) * 2.0 + 0.5, nef.Lors(lors)))
        elif kind == "autograd":
            imgs = [_phantom(case, ic, seed + b) * (1.0 + 0.1 * b) + 0.05 for b in range(case["images"])]
            x = torch.stack(imgs) if case["images"] > 1 else imgs[0]
            shape = (case["images"], n) if case["images"] > 1 else (n,)
            y = torch.poisson(_rand(seed + 4, *shape) * 8.0, generator=torch.Generator(device=_dev()).manual_seed(seed + 5))
            s.update(x=x.contiguous().requires_grad_(True), y=y,
                     tof=(sc.tof.tof_bin, sc.tof.tof_sigma2) if tof else None)
        else:  # mlem, osem: values are the attenuation correction factors of the events
            y = torch.exp(_rand(seed + 3, n) * 1.5)
            eff = sc.tof.tof_bin if tof else 80.0
            em = _sensitivity(sc, ic, n, 2.32, eff, seed + 6)
            L = 2 * sc.average_radius / ic.unit_size[0]
            add = _rand(seed + 7, n) * (20.0 * eff / L / L) if case.get("add") else None
            s.update(lm=nef.Listmode(y, nef.Lors(lors)), emap=nef.Emap(em, ic.center, ic.size), add=add)
    return s


# ------------------------------------------------------------------ one pass


def run(s):
    """One pass through the public entry points."""
    kind, case = s["kind"], s["case"]
    if kind == "project":
        return s["op"](s["image"], s["lm"].lors).data
    if kind == "backproject":
        return s["op"](s["lm"], s["image"]).data
    if kind == "mlem":
        return nef.MlemFull(case["iters"], s["ic"], s["sc"], s["lm"], None, None, None, s["emap"])().data
    if kind == "osem":
        return nef.OsemFullTof(1, case["subsets"], s["ic"], s["sc"], s["lm"], s["emap"], tof_nsigma=case["nsigma"],
                               seed=17, add=s["add"], subsets=case["order"])().data
    if kind == "autograd":
        x, ic = s["x"], s["ic"]
        x.grad = None
        p = autograd.project(x, s["lors"], ic.center, ic.size, tof=s["tof"], tof_nsigma=case["nsigma"])
        loss = autograd.poisson_nll(p, s["y"], eps=1e-3)
        loss.backward()
        return [p.detach(), x.grad]
    if kind == "emap":
        return s["gen"](s["image"]).data
    if kind == "sss":
        return scatter_sinogram.sss_sinogram(s["geo"], s["em"], s["mu"], bins=s["bins"])
    if kind == "snap":
        return s["trans"](s["lm"]).lors.data
    batch = s["batch"]
    batch.reset()
    for _ in range(case["iters"]):
        batch.replay()
    return batch.images()


# ------------------------------------------------------------------ what a pass cannot do without

# A slab of a LOR needs its two face coordinates in two axes, their floors and fractions, and on
# average 1.7 voxels; a TOF slab also its Gaussian. The figures below are operations per slab.
SLAB_FLOPS, SLAB_TOF_FLOPS, VISIT_FLOPS = 16.0, 6.0, 1.7 * 2.0


def _slabs_per_lor(case, ic, tof, nsigma):
    full = 0.7 * min(ic.shape[0], ic.shape[1])  # LORs through the body cross most of the field of view
    if not (tof and nsigma > 0):
        return full
    return min(full, 2 * nsigma * 33.7 / ic.unit_size[0] * 0.85)


def work(case):
    kind = case["kind"]
    if kind == "snap":
        return {"bytes": case["events"] * 56.0, "flops": case["events"] * 60.0}
    if kind == "sss":
        bins = case["bins"] or 827424
        crystals = 8112 if bins > 4000 else min(8112, 2 * bins)
        points = 576
        trace = crystals * points * 2 * 24.0 * (SLAB_FLOPS + VISIT_FLOPS)
        return {"bytes": 4.0 * (bins * 3 + 2 * 64 * 64 * 32 + crystals * 3), "flops": bins * points * 60.0 + trace}
    if kind == "emap":
        ic = _image_config(case)
        pairs = float(case["blocks"] * case["crystals"] ** 2 * case["rings"]) ** 2 / 2  # a pair and its reverse are one line
        slabs = 0.45 * min(ic.shape[0], ic.shape[1])
        return {"bytes": 4.0 * ic.shape[0] * ic.shape[1] * ic.shape[2], "flops": pairs * slabs * (SLAB_FLOPS + VISIT_FLOPS)}
    if kind == "studies":
        b = f = 0.0
        for shape, vox, n in _study_list(case):
            slabs = min(0.7 * shape[0], 6 * 33.7 / vox * 0.85)
            b += case["iters"] * (28.0 * n + 3 * 4 * shape[0] * shape[1] * shape[2])
            f += case["iters"] * n * slabs * (SLAB_FLOPS + SLAB_TOF_FLOPS + 2 * VISIT_FLOPS)
        return {"bytes": b, "flops": f}
    ic = _image_config(case)
    vox = float(ic.shape[0]) * ic.shape[1] * ic.shape[2]
    tof, nsigma = case.get("tof", kind == "osem"), case.get("nsigma", 0.0)
    row = 28.0 if tof else 24.0
    n = float(case["events"])
    per = _slabs_per_lor(case, ic, tof, nsigma) * n
    geo = per * (SLAB_FLOPS + (SLAB_TOF_FLOPS if tof else 0.0))
    if kind in ("project", "backproject"):
        return {"bytes": n * (row + 4) + 4 * vox, "flops": geo + per * VISIT_FLOPS}
    if kind == "autograd":
        B = case["images"]
        return {"bytes": 2 * n * row + 8 * n * B + 8 * vox * B, "flops": 2 * geo + 2 * B * per * VISIT_FLOPS}
    iters = case.get("iters", 1)
    return {"bytes": iters * n * (row + 4) + (4 * n if case.get("add") else 0) + 8 * vox,
            "flops": iters * (geo + 2 * per * VISIT_FLOPS)}


# ------------------------------------------------------------------ the same in 64 bits


def _slab_weights(l, tv, ic, dom, tof, nsigma):
    """Of LORs with one dominant transaxial axis (dom: x), per slab and voxel slot: flat voxel indices
    (m, S, 3) of an (nx, ny, nz) array and weights in mm (zero where there is no visit); per slab whether
    the projector's endpoint rule keeps it; per LOR its length in voxels and the projector's steep rule."""
    nx, ny, nz = ic.shape
    dx = ic.size[0] / nx
    dy, dz = ic.size[1] / ny / dx, ic.size[2] / nz / dx
    c = torch.tensor(list(ic.center) * 2, dtype=torch.float64, device=l.device)
    P = (l[:, :6].double() - c) / dx
    a, b = (0, 1) if dom else (1, 0)
    p1, p2, q1, q2, z1, z2 = (P[:, k, None] for k in (a, a + 3, b, b + 3, 2, 5))
    pd = p2 - p1
    kq, kz = (q2 - q1) / pd, (z2 - z1) / pd
    rt = torch.sqrt(pd ** 2 + (q2 - q1) ** 2)
    L = torch.sqrt(rt ** 2 + (z2 - z1) ** 2)
    n_p, n_q = (nx, ny) if dom else (ny, nx)
    dq, dpc = (dy, 1.0) if dom else (1.0, dy)
    S, s0 = n_p, torch.zeros_like(p1)
    if tof is not None:
        ratio = (1 - tv[:, None].double() / dx / L) / 2
        bin_ = tof[0] / dx
        expand = tof[1] / dx / dx + bin_ * bin_ / 12
        if nsigma > 0:
            hw = nsigma * math.sqrt(expand) / dpc
            if 2 * hw + 3 < n_p:
                S = int(2 * hw) + 3
                s0 = torch.floor((p1 + ratio * pd) / dpc + n_p // 2 - 0.5 - hw)
    ip = s0 + torch.arange(S, device=l.device, dtype=torch.float64)[None, :]
    wt = torch.sqrt(1 + kq ** 2 + kz ** 2) * dx * ((ip >= 0) & (ip < n_p) & (rt >= 10))
    if tof is not None:
        t2 = ((((ip - n_p // 2 + 0.5) * dpc - p1) / pd - ratio) * L) ** 2 / expand
        wt = wt * bin_ * torch.exp(-0.5 * t2) / math.sqrt(2 * float(np.float32(3.1415926)) * expand)
        if nsigma > 0:
            wt = wt * (t2 <= nsigma * nsigma)
    lo = ip - n_p / 2
    hi = lo + 1
    if tof is None:
        keep = ~(((p1 < p2) & (hi > p2)) | ((p1 >= p2) & (lo < p2)))
    elif dom:
        keep = ~(((p2 > p1) & (lo <= p1)) | ((p2 < p1) & (hi >= p1)))
    else:
        keep = ~(((p2 > p1) & (lo < p1)) | ((p2 < p1) & (hi > p1)))

    def faces(v1, k, d, half):
        u, w = (v1 + k * (lo - p1)) / d + half, (v1 + k * (hi - p1)) / d + half
        v_lo, v_hi = torch.where(k >= 0, u, w), torch.where(k >= 0, w, u)
        # a line that runs along a face (crystals and voxel faces line up on symmetric scanners) lies in
        # the upper voxel: in 64 bits its coordinate may miss the face by the rounding of the endpoints
        c1, c2 = torch.floor(v_lo + 1e-6), torch.floor(v_hi + 1e-6)
        f = torch.where(c1 != c2, (c2 - v_lo) / (v_hi - v_lo), torch.ones_like(v_lo))
        return c1, c2, f

    c1, c2, fq = faces(q1, kq, dq, n_q / 2)
    e1, e2, fz = faces(z1, kz, dz, nz / 2)
    first = fq > fz
    qm, zm = c1 >= -1, e1 >= -1
    A, B = (c1 >= 0) & (c1 < n_q), (e1 >= 0) & (e1 < nz)
    C, D = (c2 >= 0) & (c2 < n_q), (e2 >= 0) & (e2 < nz)
    w = torch.stack([torch.minimum(fq, fz) * (A & B),
                     (fq - fz).abs() * torch.where(first, A & D & zm, C & B & qm),
                     (1 - torch.maximum(fq, fz)) * (C & D & qm & zm)], 2) * wt[:, :, None]
    ipc = ip.clamp(0, n_p - 1).long()[:, :, None]
    iq = torch.stack([c1, torch.where(first, c1, c2), c2], 2).clamp(0, n_q - 1).long()
    iz = torch.stack([e1, torch.where(first, e2, e1), e2], 2).clamp(0, nz - 1).long()
    idx = ((ipc * ny + iq) if dom else (iq * ny + ipc)) * nz + iz
    steep = rt[:, 0] < (z2 - z1).abs()[:, 0]
    return idx, w, keep, L[:, 0], steep


def _trace(lors, ic, tof, nsigma, tie_x=False):
    """(rows, *_slab_weights) over all LORs in pieces. The dominant axis is decided on the float32
    endpoints in voxel units (a LOR at 45 degrees belongs to either)."""
    dx = torch.tensor(ic.size[0], dtype=torch.float32) / ic.shape[0]
    dx = dx.to(lors.device)
    d = ((lors[:, 3:5] - torch.tensor(ic.center[:2], device=lors.device)) / dx
         - (lors[:, 0:2] - torch.tensor(ic.center[:2], device=lors.device)) / dx).abs()
    xdom = (d[:, 0] >= d[:, 1]) if tie_x else (d[:, 0] > d[:, 1])
    for dom in (True, False):
        rows = torch.nonzero(xdom == dom)[:, 0]
        width = ic.shape[0] if dom else ic.shape[1]
        if tof is not None and nsigma > 0:
            width = min(width, int(2 * nsigma * math.sqrt(tof[1]) / min(ic.unit_size[:2])) + 4)
        for part in rows.split(max(1, 5000000 // width)):
            if part.numel():
                l = lors[part]
                yield (part,) + _slab_weights(l, l[:, 6] if tof is not None else None, ic, dom, tof, nsigma)


def _project64(x, lors, ic, tof, nsigma):
    """x: (nx ny nz,) or (nx ny nz, B) in 64 bits."""
    out = torch.zeros((lors.shape[0],) + tuple(x.shape[1:]), dtype=torch.float64, device=x.device)
    for rows, idx, w, keep, L, steep in _trace(lors, ic, tof, nsigma, tie_x=tof is None):
        w = w * keep[:, :, None] / (L * L)[:, None, None]
        if tof is None:
            w = w * (~steep)[:, None, None]
        if x.dim() == 1:
            out[rows] = (x[idx] * w).sum((1, 2))
        else:
            out[rows] = torch.stack([(x[:, b].contiguous()[idx] * w).sum((1, 2)) for b in range(x.shape[1])], 1)
    return out


def _backproject64(val, lors, ic, tof, nsigma, adjoint=False):
    n = ic.shape[0] * ic.shape[1] * ic.shape[2]
    acc = [torch.zeros(n, dtype=torch.float64, device=lors.device) for _ in range(val.shape[1])]
    for rows, idx, w, keep, L, steep in _trace(lors, ic, tof, nsigma, tie_x=adjoint and tof is None):
        if adjoint:
            w = w * keep[:, :, None] / (L * L)[:, None, None]
            if tof is None:
                w = w * (~steep)[:, None, None]
        for b, a in enumerate(acc):
            a.index_add_(0, idx.reshape(-1), (w * val[rows, b][:, None, None]).reshape(-1))
    return torch.stack(acc, 1)


def _em_step64(x, lors, y, add, em, ic, tof, nsigma, eps):
    """x * (A^T (y / (A x + add + eps))) / em."""
    ratio = lambda p: torch.where(p == 0, torch.zeros_like(p), y / p)  # noqa: E731
    if tof is None:
        r = ratio(_project64(x, lors, ic, None, 0.0) + eps)
        bp = _backproject64(r[:, None], lors, ic, None, 0.0)[:, 0]
    else:
        bp = torch.zeros_like(x)
        for rows, idx, w, keep, L, _ in _trace(lors, ic, tof, nsigma):
            p = (x[idx] * w * keep[:, :, None]).sum((1, 2)) / (L * L) + eps
            p = p if add is None else p + add[rows]
            r = torch.where(p == 0, torch.zeros_like(p), y[rows] / p)
            bp.index_add_(0, idx.reshape(-1), (w * r[:, None, None]).reshape(-1))
    return x * bp / torch.where(em == 0, torch.full_like(em, 1e8), em)


def _exact_sss(case, seed):
    s = prepare(case, seed)
    geo, ic = s["geo"], s["geo"].ic
    sc, sp = geo.scanner, geo.scatter_points_dev
    em, mu = s["em"].double().reshape(-1), s["mu"].double().reshape(-1)
    pairs = geo.pairs_dev if s["bins"] is None else geo.pairs_dev[s["bins"]]
    cpos = geo.vpos_dev
    m, k = cpos.shape[0], sp.shape[0]
    sumup = torch.empty(m, k, dtype=torch.float64, device=em.device)
    atten = torch.empty_like(sumup)
    both = torch.stack([em, mu], 1)
    for part in torch.arange(m, device=em.device).split(1024):
        l = torch.cat([cpos[part][:, None, :].expand(-1, k, 3), sp[None].expand(part.numel(), k, 3)], 2).reshape(-1, 6)
        p = _project64(both, l.contiguous(), ic, None, 0.0)
        d2 = ((l[:, 3:6].double() - l[:, 0:3].double()) ** 2).sum(1)
        sumup[part] = (p[:, 0] * d2).reshape(-1, k)
        atten[part] = torch.exp(-p[:, 1] * d2 / ic.unit_size[0]).reshape(-1, k)
    cp, spd = cpos.double(), sp.double()
    n_blocks, n_cr, grid1 = sc.nb_blocks_per_ring, sc.nb_blocks_per_ring * sc.blocks.shape[1], sc.blocks.shape[1]
    th = torch.rad2deg(torch.acos(cp[:, 0] / cp.norm(dim=1)))
    th = torch.where(cp[:, 1] < 0, 360 - th, th)
    th = torch.remainder(th + 180.0 / n_cr * grid1, 360.0)
    block = torch.floor(th / 360 * n_blocks) / n_blocks * 2 * math.pi
    normal = torch.stack([torch.cos(block), torch.sin(block)], 1)
    deg = torch.arange(181, dtype=torch.float64, device=em.device) / 180 * math.pi
    e_sc = 511.0 / (2 - torch.cos(deg))
    res2 = 511.0 * 0.15 ** 2
    eff = sum(torch.exp(-(e - e_sc) ** 2 / 2 / res2) for e in range(350, 650, 5))
    kn = 1 / (2 - deg) ** 2 * ((1 + deg ** 2) / 2 + (1 - deg) ** 2 / 2 / (2 - deg))
    kn = kn / (math.pi * (40 / 9 - 3 * math.log(3)))
    ge = eff * kn
    shape = mu.new_tensor([float(v) for v in ic.shape])
    g = ((spd / mu.new_tensor([float(v) for v in ic.size]) + 0.5) * shape).long()
    mu_s = mu[(g[:, 0] * ic.shape[1] + g[:, 1]) * ic.shape[2] + g[:, 2]]
    out = []
    for pr in pairs.long().split(8192):
        A, B = cp[pr[:, 0]], cp[pr[:, 1]]
        dA, dB = A[:, None, :] - spd[None], B[:, None, :] - spd[None]
        as2, sb2 = (dA ** 2).sum(2), (dB ** 2).sum(2)
        ab2 = ((A - B) ** 2).sum(1)[:, None]
        sa, sb = torch.sqrt(as2), torch.sqrt(sb2)
        arg = (-(as2 + sb2 - ab2) / (2 * sa * sb)).clamp(-1, 1)
        t = torch.floor(torch.rad2deg(torch.acos(arg))).long().clamp(0, 180)
        exp_ = 511.0 / e_sc[t]
        aA, aB, eA, eB = atten[pr[:, 0]], atten[pr[:, 1]], sumup[pr[:, 0]], sumup[pr[:, 1]]
        both_i = aA * aB ** exp_ * eA + aA ** exp_ * aB * eB
        nA, nB = normal[pr[:, 0]], normal[pr[:, 1]]
        pa = (dA[:, :, 0] * nA[:, None, 0] + dA[:, :, 1] * nA[:, None, 1]) / sa
        pb = (dB[:, :, 0] * nB[:, None, 0] + dB[:, :, 1] * nB[:, None, 1]) / sb
        out.append((pa * pb * ge[t] * mu_s[None] * both_i / as2 / sb2).sum(1))
    return torch.cat(out)


def _exact_snap(case, seed):
    s = prepare(case, seed)
    sc, raw = s["sc"], s["lors"].double()
    b, apb, half = sc.blocks, sc.angle_per_block, sc.axial_length / 2
    out = raw.clone()
    for k in range(2):
        x, y, z = raw[:, 3 * k], raw[:, 3 * k + 1], raw[:, 3 * k + 2]
        blk = torch.remainder(torch.round(torch.atan2(y, x) / apb), sc.nb_blocks_per_ring)
        ring = torch.floor((z + half) / (sc.gap + b.size[2]))
        ang = blk * apb
        iy = torch.round((-x * torch.sin(ang) + y * torch.cos(ang) + b.size[1] / 2) / b.unit_size[1] - 0.5)
        iz = torch.round((z + half - ring * (b.size[2] + sc.gap)) / b.unit_size[2] - 0.5)
        yy = (iy + 0.5) * b.unit_size[1] - b.size[1] / 2
        out[:, 3 * k] = sc.average_radius * torch.cos(ang) - yy * torch.sin(ang)
        out[:, 3 * k + 1] = sc.average_radius * torch.sin(ang) + yy * torch.cos(ang)
        out[:, 3 * k + 2] = (iz + 0.5) * b.unit_size[2] + ring * (sc.gap + b.size[2]) - half
    return out


def _exact_emap(case, seed):
    pairs = (case["blocks"] * case["crystals"] ** 2 * case["rings"]) ** 2
    if pairs * case["nx"] > 8e9:
        return None  # over 20 s
    sc, ic = _emap_scanner(case, seed), _image_config(case)
    single = sc.update(nb_blocks_per_ring=1)
    m = sc.nb_crystals_per_block * sc.nb_rings
    pos = torch.as_tensor(nef.EcatIndexToCrystalPos(single)(np.arange(m)), dtype=torch.float64, device=_dev())
    table = []
    for i in range(sc.nb_blocks_per_ring):
        a = i * sc.angle_per_block
        table.append(torch.stack([pos[:, 0] * math.cos(a) - pos[:, 1] * math.sin(a),
                                  pos[:, 0] * math.sin(a) + pos[:, 1] * math.cos(a), pos[:, 2]], 1).float())
    table = torch.cat(table)
    n = table.shape[0]
    acc = torch.zeros(ic.shape[0] * ic.shape[1] * ic.shape[2], 1, dtype=torch.float64, device=_dev())
    for part in torch.arange(n, device=_dev()).split(max(1, 4000000 // n)):
        l = torch.cat([table[part][:, None].expand(-1, n, 3), table[None].expand(part.numel(), n, 3)], 2).reshape(-1, 6)
        acc += _backproject64(torch.ones(l.shape[0], 1, dtype=torch.float64, device=_dev()), l.contiguous(), ic, None, 0.0)
    return acc.reshape(ic.shape)


def exact(case, seed):
    """What ``run`` returns for these inputs, in 64 bits, by plain torch on the inputs alone."""
    kind = case["kind"]
    if kind == "sss":
        return _exact_sss(case, seed)
    if kind == "snap":
        return _exact_snap(case, seed)
    if kind == "emap":
        return _exact_emap(case, seed)
    if kind == "studies":
        sc, inputs = _study_inputs(case, seed)
        tof, rng, out = (sc.tof.tof_bin, sc.tof.tof_sigma2), np.random.default_rng(0), []
        for ic, lors, em in inputs:
            n, per = lors.shape[0], lors.shape[0] // case["subsets"]
            lors = lors[torch.as_tensor(rng.permutation(n), device=lors.device)]
            x, e = torch.ones(em.numel(), dtype=torch.float64, device=em.device), em.double().reshape(-1)
            one = torch.ones(per, dtype=torch.float64, device=em.device)
            for _ in range(case["iters"]):
                for k in range(case["subsets"]):
                    x = _em_step64(x, lors[k * per:(k + 1) * per], one, None, e, ic, tof, 3.0, 1e-5)
            out.append(x.reshape(ic.shape))
        return out
    s = prepare(case, seed)
    ic, sc, lors = s["ic"], s["sc"], s["lors"]
    tof = (sc.tof.tof_bin, sc.tof.tof_sigma2) if case.get("tof", kind == "osem") else None
    nsigma = case.get("nsigma", 0.0)
    if kind == "project":
        return _project64(s["image"].data.double().reshape(-1), lors, ic, tof, nsigma)
    if kind == "backproject":
        return _backproject64(s["lm"].data.double()[:, None], lors, ic, tof, nsigma)[:, 0].reshape(ic.shape)
    if kind == "autograd":
        B = case["images"]
        x = s["x"].detach().double().reshape(B, -1).t().contiguous()
        y = s["y"].double().reshape(B, -1).t()
        p = _project64(x, lors, ic, tof, nsigma)
        grad = _backproject64(1 - y / (p + 1e-3), lors, ic, tof, nsigma, adjoint=True)
        p, grad = p.t(), grad.t().reshape([B] + list(ic.shape))
        return [p.contiguous(), grad.contiguous()] if B > 1 else [p[0].contiguous(), grad[0].contiguous()]
    y, em = s["lm"].data.double(), s["emap"].data.double().reshape(-1)
    x = torch.ones_like(em)
    if kind == "mlem":
        for _ in range(case["iters"]):
            x = _em_step64(x, lors, y, None, em, ic, None, 0.0, 0.0)
        return x.reshape(ic.shape)
    n, k_sub = lors.shape[0], case["subsets"]
    per = n // k_sub
    em = em / k_sub
    perm = torch.as_tensor(np.random.default_rng(17).permutation(n), device=lors.device) if case["order"] == "random" else None
    add = None if s["add"] is None else s["add"].double()
    for k in range(k_sub):
        rows = perm[k * per:(k + 1) * per] if perm is not None else slice(k, per * k_sub, k_sub)
        x = _em_step64(x, lors[rows], y[rows], None if add is None else add[rows], em, ic, tof, nsigma, 1e-5)
    return x.reshape(ic.shape)
