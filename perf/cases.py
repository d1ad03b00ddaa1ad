"""The work that a user of this package has it do, as cases that can be timed one by one.

Eight kinds of case, each through the package's public entry points:
  slices    slices of a scan that is already filtered (`reconstruct_planes_tensor`)
  volume    the whole volume of such a scan (`reconstruct_volume_tensor`)
  scan      raw detector counts into filtered views (`reset`, `add_raw_projections`), from
            device memory, or from page-locked host memory followed by slices
  live      a block of line integrals with tilt and Gaussian correction (`add_projections`)
  cor       the rotation-centre search's scores (`cor_scores`)
  gradient  a slice of the differentiable back-projector, forward and backward
  otsu      the air / bone threshold of a volume (`model.otsu_threshold`)
  surface   the iso-surface of a volume (`model.marching_cubes`)

The sizes are those of the package's benchmark and tests: a 486 x 384 detector with 600
views (cone beam), a 1944 x 1536 detector at full resolution, a 128 x 128 parallel-beam
scan, volumes of some hundred voxels a side. Scans are seeded synthetic ones: random
ellipsoids, uneven flat and dark fields, Poisson counts.
"""
import math

import numpy as np
import torch

from tomography_local_demo_b200 import ParallelGeometry, SliceReconstructor, circular_cone_vectors
from tomography_local_demo_b200 import model
from tomography_local_demo_b200 import phantom
from tomography_local_demo_b200 import recon
from tomography_local_demo_b200.autograd import BackprojectOp, backproject

SOD, SDD, WIDTH = 440.0, 680.0, 145.3           # mm: source-axis, source-detector, detector width
DEV = "cuda"
F64 = torch.float64


def listed():
    cone = dict(beam="cone", views=600, rows=384, cols=486, window="shepp-logan")
    return [
        # one slice of a small parallel-beam scan: the latency of a single interactive request
        dict(name="slice_small_parallel", kind="slices", beam="parallel", views=180, rows=128, cols=128,
             window="shepp-logan", filter="fft", store="fp32", slices=1, n=128, zoom=1.0),
        # the three oblique slices of the viewer, at its full size, from the 16-bit ring
        dict(cone, name="slices_3x512_bf16", kind="slices", filter="tc", store="bf16", slices=3, n=512, zoom=1.0),
        # a batch of zoomed slices of uneven size from full-resolution views
        dict(name="slices_full_detector", kind="slices", beam="cone", views=160, rows=1536, cols=1944,
             window="ram-lak", filter="fft", store="fp32", slices=10, n=601, zoom=2.5),
        # the volume for the threshold and the surface
        dict(cone, name="volume_256", kind="volume", filter="tc", store="bf16", maxdim=256),
        # a whole scan of raw counts on the device, through the tensor-core filter
        dict(cone, name="scan_tensor_cores", kind="scan", filter="tc", store="bf16", host=False),
        # full-resolution views through the FFT filter
        dict(name="scan_full_detector", kind="scan", beam="cone", views=96, rows=1536, cols=1944,
             window="ram-lak", filter="fft", store="fp32", host=False),
        # a scan that arrives in page-locked host memory, and its three slices
        dict(cone, name="scan_from_host", kind="scan", filter="fft", store="bf16", host=True, views=200, n=512),
        # a block of views of a live scan, with the pre-processing that the scanner needs
        dict(cone, name="live_block", kind="live", views=64, filter="fft", store="fp32", sigma=1.0, tilt=0.3),
        # the trial slices of the rotation-centre search
        dict(cone, name="cor_search", kind="cor", filter="fft", store="fp32", trials=25, n=192),
        # one step of a gradient method on a slice: loss, and gradients of views, shift and tilt
        dict(cone, name="gradient_512", kind="gradient", n=512, shift=1.7, tilt=0.3),
        # the threshold of a reconstructed volume
        dict(name="otsu_512", kind="otsu", nx=512, ny=512, nz=512, bins=512),
        # the bone surface of a reconstructed volume
        dict(name="surface_320", kind="surface", nx=320, ny=320, nz=301, noise=0.08),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the listed kinds, sizes spread over their ranges."""
    kind = rng.choice(["slices", "slices", "volume", "scan", "scan", "live", "cor", "gradient", "otsu", "surface"])
    if kind == "otsu":
        return dict(kind=kind, nx=_log(rng, 33, 512), ny=_log(rng, 33, 512), nz=_log(rng, 33, 512),
                    bins=rng.choice([128, 256, 512]))
    if kind == "surface":
        return dict(kind=kind, nx=_log(rng, 33, 320), ny=_log(rng, 33, 320), nz=_log(rng, 33, 320),
                    noise=rng.choice([0.0, 0.05, 0.1]))
    beam = "cone" if kind in ("scan", "live") else rng.choice(["cone", "cone", "parallel"])
    cols = _log(rng, 100, 1944 if kind == "scan" else 640)
    rows = max(32, int(cols * rng.uniform(0.6, 1.1)))
    views = max(8, min(_log(rng, 30, 600), 280_000_000 // (rows * cols)))
    store = rng.choice(["fp32", "bf16"])
    filt = rng.choice(["fft", "tc"]) if cols <= 512 and store == "bf16" else "fft"
    c = dict(kind=kind, beam=beam, views=views, rows=rows, cols=cols, window=rng.choice(["shepp-logan", "ram-lak"]),
             filter=filt, store=store)
    if kind == "slices":
        n = _log(rng, 64, 1024)
        return dict(c, slices=rng.randint(1, max(1, min(12, 1_500_000 // (n * n)))), n=n,
                    zoom=rng.choice([1.0, 1.7, 4.0]))
    if kind == "volume":
        return dict(c, maxdim=min(_log(rng, 40, 256), int((5e9 / views) ** (1 / 3))))
    if kind == "scan":
        host = rng.random() < 0.3
        return dict(c, host=host, n=rng.randint(100, 512)) if host else dict(c, host=False)
    if kind == "live":
        return dict(c, views=min(views, 100), sigma=rng.choice([0.0, 0.8, 1.0, 1.5]),
                    tilt=rng.choice([0.0, 0.3, -1.2]))
    if kind == "cor":
        return dict(c, trials=rng.randint(9, 33), n=rng.randint(128, 256))
    return {**{k: c[k] for k in ("kind", "beam", "views", "rows", "cols", "window")}, "n": _log(rng, 96, 512),
            "shift": round(rng.uniform(-3, 3), 2), "tilt": rng.choice([0.0, 0.3, -0.5])}


# ------------------------------------------------------------------ inputs
def _geometry(case):
    R, C = case["rows"], case["cols"]
    if case["beam"] == "parallel":
        return ParallelGeometry(np.arange(case["views"]) * np.pi / case["views"], R, C, 94.0 / C, 94.0 / C)
    return circular_cone_vectors(case["views"], SOD, SDD, R, C, WIDTH / C)


def _line_integrals(case, seed):
    """Line integrals [views, rows, cols] f32 of a dozen random ellipsoids."""
    ph = phantom.EllipsoidPhantom(1.0, phantom.random_ellipsoids(12, seed % (1 << 31), mu_range=(0.01, 0.05)))
    geom = _geometry(case)
    if case["beam"] == "parallel":
        return phantom.project_parallel_torch(ph, geom, DEV).permute(1, 0, 2).contiguous()
    return phantom.project_cone_torch(ph, geom, DEV)


def _raw_scan(case, seed):
    """(uint16 counts [views, rows, cols], flat, dark), as the detector gives them."""
    p = _line_integrals(case, seed)
    gen = torch.Generator(device=DEV)
    gen.manual_seed(seed)
    shape = p.shape[1:]
    flat = (50000.0 * (1.0 + 0.02 * torch.randn(shape, generator=gen, device=DEV))).round().clamp(1000, 65000)
    dark = (100.0 + 5.0 * torch.randn(shape, generator=gen, device=DEV)).round().clamp(0, 500)
    raw = torch.empty(p.shape, dtype=torch.int16, device=DEV)
    for v0 in range(0, len(p), 64):
        mean = (flat - dark) * torch.exp(-p[v0:v0 + 64])
        counts = (torch.poisson(mean, generator=gen) + dark).clamp(0, 65535)
        raw[v0:v0 + 64] = counts.to(torch.int32).to(torch.int16)
    return raw.view(torch.uint16), flat, dark


def _volume(case, seed):
    """Volume as the reconstruction leaves it: smooth bodies, noise, zeros outside the field of
    view. For the surface the bodies stay and the seed shades them (a smooth gain about 0.5), so
    that every seed has other vertices on the same number of edges."""
    surface = case["kind"] == "surface"
    shading, seed = seed, 7 if surface else seed
    gen = torch.Generator(device=DEV)
    gen.manual_seed(seed)
    shape = (case["nx"], case["ny"], case["nz"])
    x, y, z = (torch.linspace(-1, 1, n, device=DEV) for n in shape)
    vol = torch.empty(shape, dtype=torch.float32, device=DEV).normal_(generator=gen).mul_(case.get("noise", 0.05))
    rng = np.random.default_rng(seed)
    for _ in range(8):
        c, a, value = rng.uniform(-0.5, 0.5, 3), rng.uniform(0.12, 0.45, 3), rng.uniform(0.7, 1.0)
        q = (((x - c[0]) / a[0]) ** 2)[:, None, None] + (((y - c[1]) / a[1]) ** 2)[:, None] + ((z - c[2]) / a[2]) ** 2
        vol += value * torch.sigmoid((1.0 - q) * 20.0)
        del q
    if surface:
        px, py, pz = np.random.default_rng(shading).uniform(0, 2 * np.pi, 3)
        gain = 1.0 + 0.2 * (torch.sin(3 * x + px)[:, None, None] + torch.sin(2 * y + py)[:, None] + torch.sin(4 * z + pz))
        vol -= 0.5
        vol = torch.where(vol > 0, vol.clamp(min=1e-3), vol.clamp(max=-1e-3)) * gain + 0.5
    vol *= (x ** 2)[:, None, None] + (y ** 2)[:, None] <= 1.0
    return vol


def _requests(case, seed, count, n, zoom):
    rng = np.random.default_rng(seed + 1)
    reqs = []
    for _ in range(count):
        nrm = rng.normal(size=3)
        nrm /= np.linalg.norm(nrm)
        reqs.append(dict(origin=tuple(rng.uniform(-10, 10) * nrm), normal=tuple(nrm), n=n, zoom=zoom))
    return reqs


def _views64(case, seed):
    """Filtered views [views, rows, cols] in 64 bits, from the counts (a scan) or the line integrals."""
    if case["kind"] in ("live", "gradient"):
        x = _line_integrals(case, seed).double()
        if case["kind"] == "live":
            x = _preprocess64(x, case)
    else:
        raw, flat, dark = _raw_scan(case, seed)
        flat, dark = flat.double(), dark.double()
        x = (raw.view(torch.int16).to(torch.int32) & 0xFFFF).double()
        x = -torch.log(((x - dark) / (flat - dark).clamp(min=1.0)).clamp(min=1e-3))
    return _filter64(x, case)


# ------------------------------------------------------------------ what is measured
def _reconstructor(case, views=None):
    geom = _geometry(case if views is None else dict(case, views=views))
    return SliceReconstructor(None, geom, window=case["window"], store=case["store"], filter=case["filter"],
                              gaussian=case.get("sigma", 0.0), tilt=case.get("tilt", 0.0), verbose=False)


def prepare(case, seed):
    kind = case["kind"]
    s = dict(case=case)
    if kind in ("otsu", "surface"):
        s["volume"] = _volume(case, seed)
    elif kind == "gradient":
        geom = _geometry(case)
        R, C = case["rows"], case["cols"]
        if case["beam"] == "cone":
            maps, code = recon.cone_view_maps(recon.cone_constants(geom.vectors), R, C), 1
        else:
            maps, code = recon.parallel_view_maps(geom.angles, geom.pixel_u, geom.pixel_v, R, C), 0
        req = _requests(case, seed, 1, case["n"], 1.0)[0]
        grid = recon.plane_grid(geom.volume_box(), req["origin"], req["normal"], case["n"])
        views = torch.from_numpy(maps.view(np.uint8).copy()).to(DEV)
        s["op"] = BackprojectOp(views, code, R, C, grid.reshape(1), case["n"] ** 2)
        s["q"] = _views64(case, seed).float().contiguous().requires_grad_(True)
        s["shift"] = torch.tensor(case["shift"], requires_grad=True)
        s["tilt"] = torch.tensor(math.radians(case["tilt"]), requires_grad=True)
    elif kind == "live":
        x = _line_integrals(case, seed)
        s["rec"] = _reconstructor(case)
        s["block"] = x.permute(1, 0, 2).contiguous()
    else:
        raw, flat, dark = _raw_scan(case, seed)
        s["rec"] = rec = _reconstructor(case)
        rec.set_flat_dark(flat.cpu().numpy(), dark.cpu().numpy())
        s["requests"] = _requests(case, seed, case.get("slices", 3), case.get("n", 512), case.get("zoom", 1.0))
        if kind == "scan":
            s["raw"] = raw.cpu().pin_memory() if case["host"] else raw
        else:
            rec.add_raw_projections(np.arange(case["views"]), raw)
    torch.cuda.synchronize()
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "otsu":
        return model.otsu_threshold(s["volume"], case["bins"])
    if kind == "surface":
        return model.marching_cubes(s["volume"], 0.5, (-40.0, -40.0, -37.0), 0.25)
    if kind == "gradient":
        f = backproject(s["q"], s["shift"], s["tilt"], s["op"])
        loss = 0.5 * (f * f).sum()
        return (f.detach(),) + torch.autograd.grad(loss, (s["q"], s["shift"], s["tilt"]))
    rec = s["rec"]
    if kind == "slices":
        return rec.reconstruct_planes_tensor(s["requests"])
    if kind == "volume":
        return rec.reconstruct_volume_tensor(maxdim=case["maxdim"])[0]
    if kind == "cor":
        return rec.cor_scores(_trials(case), n=case["n"])
    rec.reset()
    if kind == "live":
        rec.add_projections(np.arange(case["views"]), s["block"])
    else:
        rec.add_raw_projections(np.arange(case["views"]), s["raw"])
        if case["host"]:
            return rec.reconstruct_planes_tensor(s["requests"])
    return rec._ring[:case["views"], :, :case["cols"]]       # the filtered views that slices are made of


def _trials(case):
    return np.linspace(-3.0, 3.0, case["trials"])


# ------------------------------------------------------------------ least work
def work(case):
    kind = case["kind"]
    if kind in ("otsu", "surface"):
        voxels = case["nx"] * case["ny"] * case["nz"]
        return {"bytes": 4 * voxels, "flops": 8 * voxels}
    pixels = case["views"] * case["rows"] * case["cols"]
    item = 2 if case.get("store") == "bf16" else 4
    fft = 2 ** math.ceil(math.log2(2 * case["cols"]))
    filtering = 5.0 * fft * math.log2(fft) * case["views"] * case["rows"]      # both directions, real rows
    if kind == "live":
        return {"bytes": (4 + item) * pixels, "flops": filtering}
    if kind == "scan":
        flops = filtering + (3 * case["n"] ** 2 * case["views"] * 26.0 if case["host"] else 0)
        return {"bytes": (2 + item) * pixels, "flops": flops}
    if kind == "gradient":
        samples = case["n"] ** 2
        return {"bytes": 8 * pixels + 8 * samples, "flops": 3 * 26.0 * samples * case["views"]}
    if kind == "volume":
        box = _geometry(case).volume_box()
        samples = int(np.prod(np.ceil(2 * box / (2 * box.max() / case["maxdim"]))))
    else:
        samples = case["n"] ** 2 * (case["trials"] if kind == "cor" else case["slices"])
    return {"bytes": item * pixels + 4 * samples, "flops": 26.0 * samples * case["views"]}


# ------------------------------------------------------------------ the same in 64 bits
def _filter64(x, case):
    """FDK / FBP row filter of line integrals [views, rows, cols]."""
    k, R, C = x.shape
    size = 2 ** math.ceil(math.log2(2 * C))
    m = np.fft.fftfreq(size, 1.0 / size).round().astype(int)
    h = np.zeros(size)
    h[0] = 0.25
    odd = m % 2 != 0
    h[odd] = -1.0 / (np.pi * m[odd]) ** 2
    H = np.real(np.fft.rfft(h))
    if case["window"] == "shepp-logan":
        H = H * np.sinc(np.fft.rfftfreq(size))
    H = torch.from_numpy(H).to(x.device)
    if case["beam"] == "cone":
        pix = WIDTH / C
        a = (torch.arange(C, dtype=F64, device=x.device) - (C - 1) / 2) * pix
        b = (torch.arange(R, dtype=F64, device=x.device) - (R - 1) / 2) * pix
        weight = SDD / torch.sqrt(SDD ** 2 + a ** 2 + (b ** 2)[:, None])
        tau = pix * SOD / SDD
    else:
        weight, tau = torch.ones((R, C), dtype=F64, device=x.device), 94.0 / C
    out = torch.empty_like(x)
    for v in range(0, k, 16):
        y = torch.fft.irfft(torch.fft.rfft(x[v:v + 16] * weight, size) * H, size)[..., :C]
        out[v:v + 16] = y / tau
    return out


def _preprocess64(x, case):
    """Rotation by -tilt (bilinear, zero outside) and the edge-padded Gaussian of [views, rows, cols]."""
    R, C = x.shape[1:]
    if case["tilt"]:
        t = math.radians(-case["tilt"])
        rr = (torch.arange(R, dtype=F64, device=x.device) - 0.5 * (R - 1))[:, None]
        cc = torch.arange(C, dtype=F64, device=x.device) - 0.5 * (C - 1)
        row = math.cos(t) * rr + math.sin(t) * cc + 0.5 * (R - 1)
        col = -math.sin(t) * rr + math.cos(t) * cc + 0.5 * (C - 1)
        x = torch.stack([_bilinear(v, row, col) for v in x])
    if case["sigma"]:
        pad = math.ceil(3 * case["sigma"])
        for axis, n in ((1, R), (2, C)):
            at = (torch.arange(-pad, n + pad, device=x.device)).clamp(0, n - 1)
            f = torch.fft.rfftfreq(n + 2 * pad, dtype=F64, device=x.device)
            g = torch.exp(-2.0 * (math.pi * f * case["sigma"]) ** 2)
            g = g[:, None] if axis == 1 else g
            y = torch.fft.irfft(torch.fft.rfft(x.index_select(axis, at), dim=axis) * g, n + 2 * pad, dim=axis)
            x = y.narrow(axis, pad, n)
    return x


def _bilinear(q, row, col):
    R, C = q.shape
    r0, c0 = torch.floor(row), torch.floor(col)
    fr, fc = row - r0, col - c0
    r0, c0 = r0.detach().clamp(-2, R + 1).long(), c0.detach().clamp(-2, C + 1).long()
    total = 0.0
    for r, wr in ((r0, 1 - fr), (r0 + 1, fr)):
        for c, wc in ((c0, 1 - fc), (c0 + 1, fc)):
            inside = (r >= 0) & (r < R) & (c >= 0) & (c < C)
            tap = q.reshape(-1).index_select(0, (r.clamp(0, R - 1) * C + c.clamp(0, C - 1)).reshape(-1)).reshape(r.shape)
            total = total + torch.where(inside, wr * wc * tap, 0.0)
    return total


def _project(case, v, pts, shift=0.0, tilt=None):
    """(row, col, weight) of points [..., 3] in view v."""
    R, C = case["rows"], case["cols"]
    x, y, z = pts.unbind(-1)
    if case["beam"] == "cone":
        a, pix = 2 * math.pi * v / case["views"], WIDTH / C
        ca, sa = math.cos(a), math.sin(a)
        depth = SOD + x * ca + y * sa
        col = SDD * (y * ca - x * sa) / depth / pix + (C - 1) / 2
        row = SDD * z / depth / pix + (R - 1) / 2
        weight = (SOD / depth) ** 2
    else:
        a, pix = math.pi * v / case["views"], 94.0 / C
        col = (y * math.cos(a) - x * math.sin(a)) / pix + (C - 1) / 2
        row = z / pix + (R - 1) / 2
        weight = torch.ones_like(x)
    if tilt is not None:
        dc, dr = col - (C - 1) / 2, row - (R - 1) / 2
        col = (C - 1) / 2 + torch.cos(tilt) * dc + torch.sin(tilt) * dr
        row = (R - 1) / 2 - torch.sin(tilt) * dc + torch.cos(tilt) * dr
    return row, col + shift, weight


def _sum_views(case, q, pts, shift=0.0, tilt=None):
    total = torch.zeros(pts.shape[:-1], dtype=F64, device=pts.device)
    for v in range(case["views"]):
        row, col, weight = _project(case, v, pts, shift, tilt)
        total += weight * _bilinear(q[v], row, col)
    return total * math.pi / case["views"]


def _plane64(box, req):
    """Points [n, n, 3] of a requested slice and which of them are inside the box."""
    n_hat = np.asarray(req["normal"]) / np.linalg.norm(req["normal"])
    up = np.array([0.0, 0.0, 1.0])
    e1 = np.cross(up, n_hat) if abs(n_hat[2]) < 0.9 else np.cross(n_hat, [0.0, 1.0, 0.0])
    e1 /= np.linalg.norm(e1)
    e2 = np.cross(n_hat, e1)
    n = req["n"]
    size = 2.0 * max(np.abs(e1) @ box, np.abs(e2) @ box) / req["zoom"]
    t = (np.arange(n) - (n - 1) / 2.0) * (size / n)
    centre = (np.asarray(req["origin"]) @ n_hat) * n_hat
    pts = centre + t[None, :, None] * e1 + t[:, None, None] * e2
    return torch.from_numpy(pts).to(DEV), torch.from_numpy(np.all(np.abs(pts) <= box, -1)).to(DEV)


def _slices64(case, q, reqs, shift=0.0, tilt=None):
    box = _geometry(case).volume_box()
    out = []
    for req in reqs:
        pts, inside = _plane64(box, req)
        out.append(torch.where(inside, _sum_views(case, q, pts, shift, tilt), 0.0))
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind == "otsu":
        return _otsu64(_volume(case, seed), case["bins"])
    if kind == "surface":
        return _vertices64(_volume(case, seed).double()), None
    q = _views64(case, seed)
    if kind == "slices" or (kind == "scan" and case["host"]):
        return _slices64(case, q, _requests(case, seed, case.get("slices", 3), case["n"], case.get("zoom", 1.0)))
    if kind in ("scan", "live"):
        return q
    if kind == "gradient":
        return _gradient64(case, q, _requests(case, seed, 1, case["n"], 1.0)[0])
    box = _geometry(case).volume_box()
    if kind == "volume":
        h = 2.0 * box.max() / case["maxdim"]
        ax = [torch.arange(int(max(math.ceil(2 * b / h), 2)), dtype=F64, device=DEV) * h - b + h / 2 for b in box]
        out = torch.empty([len(a) for a in ax], dtype=F64, device=DEV)
        for i in range(0, len(ax[0]), 64):
            pts = torch.stack(torch.meshgrid(ax[0][i:i + 64], ax[1], ax[2], indexing="ij"), -1)
            out[i:i + 64] = _sum_views(case, q, pts)
        return out
    axial = dict(origin=(0.0, 0.0, 0.0), normal=(0.0, 0.0, 1.0), n=case["n"], zoom=1.0)
    scores = []
    for shift in _trials(case):
        img = _slices64(case, q, [axial], float(shift))[0].cpu().numpy()
        hist, _ = np.histogram(img[img != 0], bins=128)
        p = hist[hist > 0] / max(hist.sum(), 1)
        scores.append(np.sum(p * np.log(p)))
    return np.array(scores)


def _gradient64(case, q, req):
    q = q.float().double()
    shift = torch.tensor(np.float32(case["shift"]), dtype=F64, device=DEV, requires_grad=True)
    tilt = torch.tensor(np.float32(math.radians(case["tilt"])), dtype=F64, device=DEV, requires_grad=True)
    with torch.no_grad():
        f = _slices64(case, q, [req], shift, tilt)[0]
    pts, inside = _plane64(_geometry(case).volume_box(), req)
    up = torch.where(inside, f, 0.0) * math.pi / case["views"]
    gq, gs, gt = torch.empty_like(q), 0.0, 0.0
    for v in range(case["views"]):
        qv = q[v].clone().requires_grad_(True)
        row, col, weight = _project(case, v, pts, shift, tilt)
        a, b, c = torch.autograd.grad((up * weight * _bilinear(qv, row, col)).sum(), (qv, shift, tilt))
        gq[v], gs, gt = a, gs + b, gt + c
    return f.reshape(-1), gq, gs, gt


def _vertices64(vol):
    """The crossing points of the grid's edges at 0.5, in the order of the edges (point, then axis)."""
    nx, ny, nz = vol.shape
    keys, points = [], []
    for axis in range(3):
        a = vol.narrow(axis, 0, vol.shape[axis] - 1)
        b = vol.narrow(axis, 1, vol.shape[axis] - 1)
        i, j, k = torch.nonzero((a > 0.5) != (b > 0.5), as_tuple=True)
        t = (0.5 - a[i, j, k]) / (b[i, j, k] - a[i, j, k])
        p = torch.stack([i, j, k], 1).double()
        p[:, axis] += t
        keys.append(((i * ny + j) * nz + k) * 3 + axis)
        points.append(p)
    p = torch.cat(points)[torch.argsort(torch.cat(keys))]
    return torch.tensor([-40.0, -40.0, -37.0], dtype=F64, device=vol.device) + 0.25 * p


def _otsu64(vol, bins):
    v = torch.sort(vol[vol != 0])[0]
    ends = []
    for percent in (0.1, 99.95):
        at = (len(v) - 1) * (percent / float(np.float32(100)))
        i = min(int(at), len(v) - 2)
        a, b = v[i].double(), v[i + 1].double()
        ends.append(float(a + (b - a) * (at - i)))
    edges = np.linspace(ends[0], ends[1], bins + 1)
    inner = torch.from_numpy(edges[1:-1]).to(v.device)
    below = torch.searchsorted(v.double(), inner, right=False).cpu().numpy()
    hist = np.diff(np.concatenate([[0], below, [len(v)]])).astype(np.float64)
    centres = 0.5 * (edges[1:] + edges[:-1])
    w0 = np.cumsum(hist)
    w1 = w0[-1] - w0
    m0 = np.cumsum(hist * centres) / np.maximum(w0, 1)
    m1 = (np.sum(hist * centres) - np.cumsum(hist * centres)) / np.maximum(w1, 1)
    return float(centres[int(np.argmax(w0 * w1 * (m0 - m1) ** 2))])
