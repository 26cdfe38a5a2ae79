"""The calls that a user of the reconstructor makes, as cases whose time and outputs are measured.

The ranges: single views to whole scans, detectors of 48 to 4000 columns (the row filter's lengths 64 to
4096), volumes of 32^3 to 2048 x 2048 slab pairs, FP32_EXACT, FP32 and MIXED, every output layout of the
filter, general (tilted) geometry, and the learned row filter in inference and in training.  Each kind of
case calls one public entry point the way its user does:

  filter   FilterEngine.run_device: the batch filter in front of any backprojection
  rows     filter_row_real32: the cuFFT-plugin drop-in, synchronous
  recon    Reconstructor: a scan from pinned host memory to a volume in pinned host memory
  bp       BackProjectionFDK on filtered device views, up to 128 per call (32 for FP32_EXACT)
  rtk      the RTK drop-in on device views, tilted geometry
  project  the ray-marching forward projector
  denoise  one sparse-view scan through the filter, the learned row filter and the backprojection
  train    one training step of the learned filter: phantom, forward, loss, adjoint, backward, Adam

Scans are SOD 1000 mm, SID 1500 mm.  fov "matched" is the benchmark geometries' own pitch (a 256 mm volume
under a 384 mm detector); "covered" widens the detector until the whole volume projects inside it, as a
scan without truncation has it.
"""
import ctypes
import math

import numpy as np
import torch

import fdk_b200 as F
from fdk_b200 import learned
from fdk_b200._lib import check, lib
from fdk_b200.backprojection import rtk_backproject_device

DEV = "cuda"
LAYOUTS = {"rows": F.LAYOUT_ROWS, "transposed": F.LAYOUT_TRANSPOSED, "mirror": F.LAYOUT_MIRROR}


def listed():
    return [
        # one view of the reference's default detector (608 x 616), as its FilterThread filters them one by one
        dict(name="filter_one_view", kind="filter", nu=608, nv=616, views=1, layout="transposed", half=False),
        # 32 views of 2048^2 into the FP32 backprojection's layout: the streaming granularity of a large scan
        dict(name="filter_2048_mirror", kind="filter", nu=2048, nv=2048, views=32, layout="mirror", half=False),
        # a pipeline that switched its cuFFT plugin: 48 views of 1536 x 1024 per call
        dict(name="rows_1536", kind="rows", nu=1536, nv=1024, views=48),
        # a preview of a few views on a coarse grid: what a call costs when there is little to do
        dict(name="recon_preview", kind="recon", nx=64, ny=64, nz=64, nu=96, nv=80, views=60, precision="mixed",
             fov="covered", batch=32),
        # a whole 256^3 scan, mixed precision, host memory to host memory
        dict(name="recon_256_mixed", kind="recon", nx=256, ny=256, nz=256, nu=256, nv=256, views=256,
             precision="mixed", fov="matched", batch=128),
        # a whole 512^3 scan in FP32
        dict(name="recon_512_fp32", kind="recon", nx=512, ny=512, nz=512, nu=512, nv=512, views=512,
             precision="fp32", fov="covered", batch=512),
        # a rank's slab pair of a 2048^3 volume: one batch of filtered views that another stage left on the device
        dict(name="bp_2048_mixed", kind="bp", nx=2048, ny=2048, nz=2048, slab=64, nu=2048, nv=2048, views=64,
             precision="mixed", fov="covered"),
        # the BackProjectionFDK drop-in at its default precision, 32 views a call
        dict(name="bp_512_exact", kind="bp", nx=512, ny=512, nz=512, slab=256, nu=608, nv=616, views=96,
             precision="fp32_exact", fov="covered"),
        # the RTK filter's call on a tilted trajectory, a volume that is no power of two
        dict(name="rtk_400_tilted", kind="rtk", nx=400, ny=384, nz=360, nu=512, nv=480, views=32, tilt=4.0),
        # projections of a 256^3 volume for 90 views of 256^2: the learned filter's training data
        dict(name="project_256", kind="project", nx=256, ny=256, nz=256, nu=256, nv=256, views=90),
        # a 90-view scan reconstructed through the learned filter
        dict(name="denoise_256", kind="denoise", nx=256, ny=256, nz=256, nu=256, nv=256, views=90),
        # one step of its training
        dict(name="train_256", kind="train", nx=256, ny=256, nz=256, nu=256, nv=256, views=90),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["filter", "filter", "rows", "recon", "bp", "bp", "rtk", "project", "denoise", "train"])
    if kind in ("filter", "rows"):
        nu, nv = _log_int(rng, 48, 4000), _log_int(rng, 24, 2400)
        views = max(1, min(_log_int(rng, 1, 96), (1 << 26) // (nu * nv)))
        if kind == "rows":
            return dict(kind=kind, nu=nu, nv=nv, views=views)
        layout = rng.choice(sorted(LAYOUTS))
        if layout == "mirror" and rng.random() < 0.7:
            nv = max(8, nv & ~7)  # the backprojection's own sizes, most of the time
        return dict(kind=kind, nu=nu, nv=nv, views=views, layout=layout, half=rng.random() < 0.3)
    if kind == "recon":
        nx, ny, nz = (_log_int(rng, 32, 320) for _ in range(3))
        precision = rng.choice(["mixed", "fp32"])
        nv = 4 * _log_int(rng, 10, 100)
        nu = rng.choice([_log_int(rng, 48, 512), 256])
        return dict(kind=kind, nx=nx, ny=ny, nz=2 * max(16, nz // 2), nu=nu, nv=128 * max(1, nv // 128) if nu == 256 else nv,
                    views=_log_int(rng, 16, 400), precision=precision,
                    fov=rng.choice(["covered", "matched"]) if precision == "mixed" else "covered",
                    batch=rng.choice([32, 128, 256]))
    if kind == "bp":
        precision = rng.choice(["fp32_exact", "fp32", "mixed"])
        nx, ny, nz = (_log_int(rng, 48, 640) for _ in range(3))
        nz = 2 * max(16, nz // 2)
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, slab=max(8, int(nz * rng.uniform(0.1, 0.5))), nu=_log_int(rng, 96, 900),
                    nv=4 * _log_int(rng, 20, 200), views=_log_int(rng, 8, 96), precision=precision, fov="covered")
    if kind == "rtk":
        nx, ny, nz = (_log_int(rng, 40, 420) for _ in range(3))
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, nu=4 * _log_int(rng, 20, 160), nv=_log_int(rng, 60, 640),
                    views=_log_int(rng, 4, 64), tilt=rng.choice([0.0, rng.uniform(0.5, 10.0)]))
    if kind == "project":
        nx, ny, nz = (_log_int(rng, 40, 280) for _ in range(3))
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, nu=_log_int(rng, 40, 300), nv=_log_int(rng, 40, 300),
                    views=_log_int(rng, 2, 60))
    n = 4 * _log_int(rng, 10, 56)
    return dict(kind=kind, nx=n, ny=n, nz=n, nu=_log_int(rng, 64, 256), nv=4 * _log_int(rng, 12, 56),
                views=_log_int(rng, 12, 90))


# ------------------------------------------------------------------------------------------------ geometry
def _param(c):
    """The scan of a case.  filter and rows cases have no volume of their own: any will do."""
    nx, ny, nz = c.get("nx", 64), c.get("ny", 64), c.get("nz", 64)
    p = F.config("c1")
    p.nx, p.ny, p.nz, p.nu, p.nv, p.nProj = nx, ny, nz, c["nu"], c["nv"], c["views"]
    p.dx = p.dy = p.dz = 256.0 / max(nx, ny, nz)
    if c.get("fov", "matched") == "matched" and c["kind"] != "rtk":
        p.du = p.dv = 384.0 / p.nu
    else:
        r = 0.5 * math.hypot(nx, ny) * p.dx
        half_u = p.SID * r / math.sqrt(p.SOD ** 2 - r ** 2)
        half_v = p.SID * 0.5 * nz * p.dz / (p.SOD - r)
        slack = 1.15 if c["kind"] == "rtk" else 1.0
        p.du, p.dv = 2 * slack * half_u / (p.nu - 5), 2 * slack * half_v / (p.nv - 5)
    return p


def _angles64(p):
    return np.array([p.direction * (i * p.scan_angle / p.nProj) / 180.0 * math.pi + p.volume_postion_angle
                     for i in range(p.nProj)])


def _mats64(p):
    """3 x 4 matrices: voxel index -> (u w, v w, w)."""
    out = []
    for a in _angles64(p):
        c, s = math.cos(a), math.sin(a)
        cx, cy, cz = (p.nx - 1) / 2, (p.ny - 1) / 2, (p.nz - 1) / 2
        xr = np.array([c * p.dx, s * p.dy, 0, -c * p.dx * cx - s * p.dy * cy])
        zc = np.array([s * p.dx, -c * p.dy, 0, -s * p.dx * cx + c * p.dy * cy + p.SOD])
        yc = np.array([0, 0, p.dz, -p.dz * cz])
        out.append(np.stack([p.SID / p.du * xr + (p.nu - 1) / 2 * zc, p.SID / p.dv * yc + (p.nv - 1) / 2 * zc, zc]))
    return np.stack(out)


def _tilted(p, degrees):
    """The orbit's matrices for a volume that leans `degrees` about its x axis."""
    t = math.radians(degrees)
    c = np.array([(p.nx - 1) / 2, (p.ny - 1) / 2, (p.nz - 1) / 2])
    rot = np.array([[1, 0, 0], [0, math.cos(t), -math.sin(t)], [0, math.sin(t), math.cos(t)]])
    a = np.eye(4)
    a[:3, :3], a[:3, 3] = rot, c - rot @ c
    return (_mats64(p) @ a).astype(np.float32).reshape(p.nProj, 12)


def _aaf(p):
    return 1.0 / 2.0 / p.du * (2.0 * math.pi / p.nProj) / 2.0 * (p.SID / p.SOD)


def _cos64(p):
    u = (np.arange(p.nu) - (p.nu - 1) / 2) * p.du
    v = ((p.nv - 1) / 2 - np.arange(p.nv)) * p.dv
    return p.SID / np.sqrt(u[None, :] ** 2 + v[:, None] ** 2 + p.SID ** 2) * p.SOD ** 2 * _aaf(p)


def _hann64(nu):
    """The ramp with its Hann window, W = the power of two above nu."""
    w = 1 << int(nu).bit_length()
    k = np.arange(w // 2 + 1)
    r = 2.0 * k / w * (1 + np.cos(2 * math.pi * k / w)) / 2
    return np.concatenate([r, r[1:-1][::-1]])


# ------------------------------------------------------------------------------------------------ inputs
def _rng(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return g


def _balls(p, seed, n=8):
    """Centres (mm), radii and densities of balls inside the volume."""
    rng = np.random.default_rng(seed)
    half = 0.5 * min(p.nx, p.ny, p.nz) * p.dx
    d = rng.normal(size=(n, 3))
    centre = d / np.linalg.norm(d, axis=1, keepdims=True) * (0.55 * half * rng.uniform(size=(n, 1)) ** (1 / 3))
    return centre, half * rng.uniform(0.08, 0.4, n), rng.uniform(-0.2, 1.0, n)


def _views(p, seed):
    """Line integrals through the balls with a little detector noise: (views, nv, nu) float32."""
    centre, radius, rho = _balls(p, seed)
    g = _rng(seed)
    u = (torch.arange(p.nu, device=DEV, dtype=torch.float32) - (p.nu - 1) / 2) * p.du
    v = (torch.arange(p.nv, device=DEV, dtype=torch.float32) - (p.nv - 1) / 2) * p.dv
    out = torch.empty((p.nProj, p.nv, p.nu), device=DEV)
    norm2 = u[None, :] ** 2 + v[:, None] ** 2 + p.SID ** 2
    ang = _angles64(p)
    step = max(1, (1 << 25) // (p.nu * p.nv))
    for i in range(0, p.nProj, step):
        a = ang[i:i + step]
        img = out[i:i + step]
        img.normal_(0.0, 0.2, generator=g)
        for (x, y, z), r, d in zip(centre, radius, rho):
            qx = torch.tensor(np.cos(a) * x - np.sin(a) * y, device=DEV, dtype=torch.float32)[:, None, None]
            qy = torch.tensor(np.sin(a) * x + np.cos(a) * y + p.SOD, device=DEV, dtype=torch.float32)[:, None, None]
            dot = qx * u[None, None, :] + qy * p.SID - z * v[None, :, None]
            dist2 = qx ** 2 + qy ** 2 + z * z - dot * dot / norm2[None]
            img += (2 * d) * (r * r - dist2).clamp_(min=0).sqrt_()
    return out


def _filtered(p, seed):
    """Filtered views in line-integral units, (views, nv, nu) float32: a stand-in for the filter's output."""
    x = _views(p, seed)
    w = 1 << int(p.nu).bit_length()
    h = torch.tensor(_hann64(p.nu)[:w // 2 + 1], device=DEV, dtype=torch.float32)
    step = max(1, (1 << 25) // (w * p.nv))
    for i in range(0, p.nProj, step):
        x[i:i + step] = torch.fft.irfft(torch.fft.rfft(x[i:i + step], n=w) * h, n=w)[..., :p.nu]
    return x


def _transposed(x):
    return x.transpose(1, 2).contiguous()


def _mirror(x, dtype):
    """(views, nv, nu) -> (views, nu, nv, 2): the values of detector rows v and nv-1-v."""
    return torch.stack([x.to(dtype), x.flip(1).to(dtype)], -1).transpose(1, 2).contiguous()


def _volume(p, seed):
    """The balls with soft edges on the voxel grid, [z][y][x]."""
    centre, radius, rho = _balls(p, seed)
    z, y, x = (torch.arange(n, device=DEV, dtype=torch.float32) for n in (p.nz, p.ny, p.nx))
    z, y, x = -(z - (p.nz - 1) / 2) * p.dz, -(y - (p.ny - 1) / 2) * p.dy, (x - (p.nx - 1) / 2) * p.dx
    out = torch.zeros((p.nz, p.ny, p.nx), device=DEV)
    for (cx, cy, cz), r, d in zip(centre, radius, rho):
        dist = ((z[:, None, None] - cz) ** 2 + (y[None, :, None] - cy) ** 2 + (x[None, None, :] - cx) ** 2).sqrt()
        out += float(d) * ((r - dist) / (2 * p.dx) + 0.5).clamp(0, 1)
    return out


def _ellipsoids(p, seed):
    """A training phantom: 20 upright ellipsoids as fdk_voxelize takes them."""
    rng = np.random.default_rng(seed)
    half = 0.5 * p.nx * p.dx
    e = np.zeros((20, 16))
    d = rng.normal(size=(20, 3))
    e[:, :3] = d / np.linalg.norm(d, axis=1, keepdims=True) * (0.8 * half * rng.uniform(size=(20, 1)) ** (1 / 3))
    e[:, 3:6] = rng.uniform(0.05, 0.4, (20, 3)) * half
    e[:, 6] = e[:, 10] = e[:, 14] = 1.0
    e[:, 15] = rng.uniform(-0.2, 1.0, 20)
    return e


def _weights(seed):
    """A network some way into its training: every layer away from zero, the output a small correction."""
    rng = np.random.default_rng(seed + 5)
    w = learned.init_params(seed).astype(np.float64)
    w[-289:-1] = rng.standard_normal(288) * 0.004
    for at, n in ((288, 32), (288 + 32 + 9216, 32)):
        w[at:at + n] = rng.standard_normal(n) * 0.01
    return w.astype(np.float32)


def _pinned(shape):
    return torch.empty(shape, dtype=torch.float32, pin_memory=True)


def _scaled_rows(p, seed):
    """Ramp-filtered detector rows in the reconstruction's units, as the learned filter reads them."""
    return (_filtered(p, seed) * (p.SOD ** 2 * _aaf(p))).contiguous()


class _Device:
    """Device memory of a library handle, for torch.as_tensor; a tensor made from it keeps the handle open."""

    def __init__(self, owner, ptr, shape):
        self.owner = owner
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": shape, "typestr": "<f4", "version": 2}


def _boxes(c, p):
    top_z = p.nz // 2 - c["slab"]
    return F.BoxT(0, 0, top_z, p.nx, p.ny, c["slab"]), F.BoxT(0, 0, p.nz // 2, p.nx, p.ny, c["slab"])


def prepare(case, seed):
    c, p = case, _param(case)
    kind = c["kind"]
    s = {"c": c, "p": p}
    if kind == "filter":
        s["engine"] = F.FilterEngine(_cos64(p).astype(np.float32), _hann64(p.nu).astype(np.float32))
        s["src"] = _views(p, seed)
        shape = {"rows": (p.nProj, p.nv, p.nu), "transposed": (p.nProj, p.nu, p.nv), "mirror": (p.nProj, p.nu, p.nv, 2)}
        s["dst"] = torch.zeros(shape[c["layout"]], device=DEV, dtype=torch.float16 if c["half"] else torch.float32)
        s["scale"] = 1.0 / (p.SOD ** 2 * _aaf(p)) if c["half"] else 1.0
    elif kind == "rows":
        s["src"] = _views(p, seed)
        s["dst"] = torch.zeros_like(s["src"])
        s["filter"] = torch.tensor(_hann64(p.nu), device=DEV, dtype=torch.float32)
    elif kind == "recon":
        s["recon"] = F.Reconstructor(p, c["precision"], batch=c["batch"])
        s["views"] = _pinned((p.nProj, p.nv, p.nu))
        s["views"].copy_(_views(p, seed))
        s["out"] = _pinned((p.nx * p.ny * p.nz,))
    elif kind == "bp":
        x = _filtered(p, seed)
        exact = c["precision"] == "fp32_exact"
        s["views"] = _transposed(x) if exact else _mirror(x, torch.float16 if c["precision"] == "mixed" else torch.float32)
        s["mats"] = p.proj_matrices()
        s["bp"] = F.BackProjectionFDK(p.nv, p.nu, 1, p.nx, p.ny, p.nz, *_boxes(c, p), c["precision"])
    elif kind == "rtk":
        s["views"] = _filtered(p, seed)
        s["mats"] = _tilted(p, c["tilt"])
        s["in"] = torch.zeros((p.nz, p.ny, p.nx), device=DEV)
        s["out"] = torch.empty_like(s["in"])
    elif kind == "project":
        s["vol"], s["g"] = _volume(p, seed), p.to_c()
        s["out"] = torch.empty((p.nProj, p.nv, p.nu), device=DEV)
    else:
        s["pipe"] = learned.Pipeline(p)
        s["w"] = torch.from_numpy(_weights(seed)).to(DEV)
        if kind == "denoise":
            s["raw"] = _views(p, seed)
            s["rows"] = torch.empty_like(s["raw"])
        else:
            s["rows"] = _scaled_rows(p, seed)
            s["ell"] = _ellipsoids(p, seed)
            s["m"] = torch.empty_like(s["w"]).normal_(0.0, 1e-6, generator=_rng(seed))
            s["v"] = torch.full_like(s["w"], 1e-8)
            s["step"] = 1000
    return s


def run(s):
    c, p = s["c"], s["p"]
    kind = c["kind"]
    if kind == "filter":
        s["engine"].run_device(s["src"].data_ptr(), s["dst"].data_ptr(), p.nProj, LAYOUTS[c["layout"]],
                               F.DTYPE_F16 if c["half"] else F.DTYPE_F32, s["scale"])
        return s["dst"]
    if kind == "rows":
        F.filter_row_real32(s["src"], s["dst"], s["filter"])
        return s["dst"]
    if kind == "recon":
        r = s["recon"]
        r.reset()
        r.push(s["views"].numpy(), 0)
        return r.volume(s["out"].numpy())
    if kind == "bp":
        bp, exact = s["bp"], c["precision"] == "fp32_exact"
        bp.reset()
        step = 32 if exact else 128
        for i in range(0, p.nProj, step):
            n = min(step, p.nProj - i)
            bp.BP_device(s["views"][i:i + n].data_ptr(), F.LAYOUT_TRANSPOSED if exact else F.LAYOUT_MIRROR,
                         s["mats"][i:i + n], n)
        ptr, _ = bp.volume_device()
        return torch.as_tensor(_Device(bp, ptr, (p.nx, p.ny, 2 * c["slab"])), device=DEV)
    if kind == "rtk":
        rtk_backproject_device((p.nu, p.nv, p.nProj), (p.nx, p.ny, p.nz), s["mats"], s["in"].data_ptr(),
                               s["out"].data_ptr(), s["views"].data_ptr())
        return s["out"]
    if kind == "project":
        check(lib().fdk_forward_project(ctypes.byref(s["g"]), s["vol"].data_ptr(), 0, p.nProj, s["out"].data_ptr(), None))
        return s["out"]
    pl, w = s["pipe"], s["w"]
    if kind == "denoise":
        pl.engine.run_device(s["raw"].data_ptr(), s["rows"].data_ptr(), p.nProj, F.LAYOUT_ROWS)
        pl.reconstruct(w, s["rows"])
        ptr, _ = pl.bp.volume_device()
        return {"rows": pl.y, "volume": torch.as_tensor(_Device(pl.bp, ptr, (p.nx, p.ny, p.nz)), device=DEV)}
    e = s["ell"]
    check(lib().fdk_voxelize(ctypes.byref(pl.g), e.ctypes.data, len(e), pl.truth.data_ptr(), None))
    pl.reconstruct(w, s["rows"])
    loss = pl.mse(with_grad=True)
    pl.gradient(w, s["rows"])
    s["step"] += 1
    check(lib().fdk_adam_step(w.data_ptr(), pl.dparams.data_ptr(), s["m"].data_ptr(), s["v"].data_ptr(), w.numel(),
                              1e-3, 0.9, 0.999, 1e-8, s["step"], None))
    return {"loss": loss, "residual": pl.res, "gradient": pl.dparams, "weights": w, "m": s["m"], "v": s["v"]}


def work(case):
    c = case
    pix = c["views"] * c["nu"] * c["nv"]
    w = 1 << int(c["nu"]).bit_length()
    fft = c["views"] * c["nv"] * 5.0 * w * math.log2(w)  # a real transform there and back
    if c["kind"] in ("filter", "rows"):
        out = pix * (2 if c.get("half") else 4) * (2 if c.get("layout") == "mirror" else 1)
        return {"bytes": 4 * pix + out, "flops": fft}
    vox = c["nx"] * c["ny"] * (2 * c["slab"] if c["kind"] == "bp" else c["nz"])
    update = 10.0 * vox * c["views"]  # a bilinear sample (3 lerps), its weight and the sum
    if c["kind"] == "recon":
        return {"bytes": 4 * pix + 4 * vox, "flops": fft + update}
    if c["kind"] == "bp":
        return {"bytes": pix * {"fp32_exact": 4, "fp32": 8, "mixed": 4}[c["precision"]] + 4 * vox, "flops": update}
    if c["kind"] == "rtk":
        return {"bytes": 4 * pix + 8 * vox, "flops": update}
    if c["kind"] == "project":
        n = 0.7 * min(c["nx"], c["ny"], c["nz"])  # samples a ray, about
        return {"bytes": 4 * pix + 4 * vox, "flops": 20.0 * pix * n}
    net = 2.0 * 9 * (32 + 32 * 32 + 32) * pix
    if c["kind"] == "denoise":
        return {"bytes": 4 * pix + 8 * pix + 4 * vox, "flops": fft + net + update}
    return {"bytes": 4 * pix + 8 * vox, "flops": 3 * net + 2 * update}


# ------------------------------------------------------------------------------------------------ in 64 bits
def _filter64(x, h, cos, pad):
    """(views, nv, nu) float64: weight, pad with the mean of the edge samples, filter, crop."""
    w, nu = len(h), x.shape[-1]
    off = (w - nu) >> 1
    h = torch.tensor(np.asarray(h, np.float64)[:w // 2 + 1], device=DEV)
    out = torch.empty(x.shape, device=DEV, dtype=torch.float64)
    step = max(1, (1 << 25) // (w * x.shape[1]))
    for i in range(0, x.shape[0], step):
        y = x[i:i + step].double()
        if cos is not None:
            y = y * torch.as_tensor(cos, device=DEV, dtype=torch.float64)
        full = torch.empty(y.shape[:-1] + (w,), device=DEV, dtype=torch.float64)
        full[..., :off] = y[..., :pad].mean(-1, keepdim=True)
        full[..., off + nu:] = y[..., nu - pad:].mean(-1, keepdim=True)
        full[..., off:off + nu] = y
        out[i:i + step] = torch.fft.irfft(torch.fft.rfft(full) * h, n=w)[..., off:off + nu]
    return out


def _sampler(m, p, zs):
    """For one view: the detector position of every voxel [zs, y, x] as grid_sample takes it, and its weight, zero
    outside the detector."""
    x, y = (torch.arange(n, device=DEV, dtype=torch.float64) for n in (p.nx, p.ny))
    z = torch.as_tensor(zs, device=DEV, dtype=torch.float64)[:, None, None]
    m = [float(t) for t in np.asarray(m, np.float64).reshape(12)]
    if m[2] == 0 and m[10] == 0:
        w = (m[8] * x[None, :] + m[9] * y[:, None] + m[11])[None]
        u = ((m[0] * x[None, :] + m[1] * y[:, None] + m[3])[None] / w).expand(len(zs), p.ny, p.nx)
    else:
        w = m[8] * x + m[9] * y[:, None] + m[10] * z + m[11]
        u = (m[0] * x + m[1] * y[:, None] + m[2] * z + m[3]) / w
    v = (m[4] * x + m[5] * y[:, None] + m[6] * z + m[7]) / w
    ok = (u >= 0) & (u < p.nu - 1) & (v >= 0) & (v < p.nv - 1)
    grid = torch.stack([u * (2 / (p.nu - 1)) - 1, v * (2 / (p.nv - 1)) - 1], -1)
    return grid.reshape(1, len(zs) * p.ny, p.nx, 2), ok / (w * w)


def _backproject64(rows, mats, p, zs):
    """rows: (views, nv, nu) float64 -> [zs, y, x]."""
    vol = torch.zeros((len(zs), p.ny, p.nx), device=DEV, dtype=torch.float64)
    part = max(1, (1 << 27) // (p.nx * p.ny))
    for a in range(0, len(zs), part):
        z = zs[a:a + part]
        for i in range(len(mats)):
            grid, weight = _sampler(mats[i], p, z)
            r = torch.nn.functional.grid_sample(rows[i][None, None], grid, align_corners=True)
            vol[a:a + part] += r.reshape(weight.shape[0], p.ny, p.nx) * weight
    return vol


def _network64(w, x, s):
    """y = x + net(s x) / s with activations held in BF16, (rows, nu) float64."""
    def held(a):
        return a + (a.detach().bfloat16().double() - a.detach())

    w1, b1, w2, b2, w3, b3 = torch.split(w, [288, 32, 9216, 32, 288, 1])
    conv = torch.nn.functional.conv1d
    a1 = held(torch.relu(conv(s * x[:, None], w1.reshape(32, 1, 9), b1, padding=4)))
    a2 = held(torch.relu(conv(a1, w2.reshape(32, 32, 9), b2, padding=4)))
    return x + conv(a2, w3.reshape(1, 32, 9), b3, padding=4)[:, 0] / s


def _project64(vol, p):
    vol = vol.double()
    half = [(p.nx - 1) / 2 * p.dx, (p.ny - 1) / 2 * p.dy, (p.nz - 1) / 2 * p.dz]
    u = (torch.arange(p.nu, device=DEV, dtype=torch.float64) - (p.nu - 1) / 2) * p.du
    v = ((p.nv - 1) / 2 - torch.arange(p.nv, device=DEV, dtype=torch.float64)) * p.dv
    out = torch.zeros((p.nProj, p.nv, p.nu), device=DEV, dtype=torch.float64)
    step = min(p.dx, p.dy, p.dz)
    flat = vol.reshape(-1)
    for i, ang in enumerate(_angles64(p)):
        c, s = math.cos(-ang), math.sin(-ang)
        far = p.SID - p.SOD
        o = (p.SOD * s, -p.SOD * c, 0.0)
        d = torch.stack([(u * c - far * s).expand(p.nv, p.nu), (u * s + far * c).expand(p.nv, p.nu),
                         v[:, None].expand(p.nv, p.nu)]) - torch.tensor(o, device=DEV, dtype=torch.float64)[:, None, None]
        d = d / d.square().sum(0).sqrt()
        t0 = torch.stack([torch.minimum((-h - q) / e, (h - q) / e) for h, q, e in zip(half, o, d)]).amax(0)
        t1 = torch.stack([torch.maximum((-h - q) / e, (h - q) / e) for h, q, e in zip(half, o, d)]).amin(0)
        count = int(((t1 - t0).max() / step).clamp(min=0).item()) + 2
        k = torch.arange(count, device=DEV, dtype=torch.float64)[:, None, None]
        t = t0 + k * step
        live = t < t1
        pos = [o[0] / p.dx + (p.nx - 1) / 2 + d[0] / p.dx * t, (p.ny - 1) / 2 - (o[1] + d[1] * t) / p.dy,
               (p.nz - 1) / 2 - (o[2] + d[2] * t) / p.dz]
        at = [q.trunc() for q in pos]
        fr = [q - a for q, a in zip(pos, at)]
        total = torch.zeros_like(t)
        for dx in (0, 1):
            for dy in (0, 1):
                for dz in (0, 1):
                    x, y, z = ((a + e).long().clamp(0, n - 1) for a, e, n in zip(at, (dx, dy, dz), (p.nx, p.ny, p.nz)))
                    wt = 1.0
                    for f, e in zip(fr, (dx, dy, dz)):
                        wt = wt * (f if e else 1 - f)
                    total += flat[(z * p.ny + y) * p.nx + x] * wt
        out[i] = (total * live).sum(0) * step
    return out


def _voxelize64(p, ell):
    z, y, x = (torch.arange(n, device=DEV, dtype=torch.float64) for n in (p.nz, p.ny, p.nx))
    z, y, x = -(z - (p.nz - 1) / 2) * p.dz, -(y - (p.ny - 1) / 2) * p.dy, (x - (p.nx - 1) / 2) * p.dx
    out = torch.zeros((p.nz, p.ny, p.nx), device=DEV, dtype=torch.float64)
    for e in ell:
        q = (((x - e[0]) / e[3]) ** 2)[None, None] + (((y - e[1]) / e[4]) ** 2)[None, :, None] + \
            (((z - e[2]) / e[5]) ** 2)[:, None, None]
        out += (q <= 1.0) * float(e[15])
    return out


def exact(case, seed):
    c, p = case, _param(case)
    kind = c["kind"]
    if kind in ("filter", "rows"):
        x = _views(p, seed)
        h = _hann64(p.nu).astype(np.float32)
        if kind == "rows":
            return _filter64(x, h, None, 3)
        y = _filter64(x, h, _cos64(p).astype(np.float32), 4)
        if c["half"]:
            y *= float(np.float32(1.0 / (p.SOD ** 2 * _aaf(p))))
        return {"rows": lambda: y, "transposed": lambda: _transposed(y), "mirror": lambda: _mirror(y, torch.float64)}[c["layout"]]()
    if kind == "recon":
        rows = _filter64(_views(p, seed), _hann64(p.nu), _cos64(p), 4)
        return _backproject64(rows, _mats64(p), p, list(range(p.nz))).cpu().numpy()
    if kind == "bp":
        x = _filtered(p, seed)
        rows = (x.half() if c["precision"] == "mixed" else x).double()
        zs = list(range(p.nz // 2 - c["slab"], p.nz // 2 + c["slab"]))
        return _backproject64(rows, p.proj_matrices(), p, zs).permute(2, 1, 0).contiguous()
    if kind == "rtk":
        return _backproject64(_filtered(p, seed).double(), _tilted(p, c["tilt"]), p, list(range(p.nz)))
    if kind == "project":
        return _project64(_volume(p, seed), p)
    s = 1.0 / (p.SOD ** 2 * _aaf(p))
    mats, zs = p.proj_matrices(), list(range(p.nz))
    w = torch.from_numpy(_weights(seed)).to(DEV).double().requires_grad_(kind == "train")
    if kind == "denoise":
        rows = _filter64(_views(p, seed), _hann64(p.nu).astype(np.float32), _cos64(p).astype(np.float32), 4)
        y = torch.cat([_network64(w, r, s) for r in rows.reshape(-1, p.nu).split(2048)]).reshape(rows.shape)
        return {"rows": y, "volume": _backproject64(y, mats, p, zs).permute(2, 1, 0).contiguous()}
    x = _scaled_rows(p, seed).double()
    with torch.no_grad():
        y = torch.cat([_network64(w, r, s) for r in x.reshape(-1, p.nu).split(2048)]).reshape(x.shape)
        diff = _backproject64(y, mats, p, zs) - _voxelize64(p, _ellipsoids(p, seed))
    n = diff.numel()
    residual = 2 * diff / n
    back = torch.empty_like(y)
    for i in range(p.nProj):
        grid, weight = _sampler(mats[i], p, zs)
        row = y[i][None, None].clone().requires_grad_(True)
        r = torch.nn.functional.grid_sample(row, grid, align_corners=True)
        back[i] = torch.autograd.grad(r, row, (residual * weight).reshape(r.shape))[0][0, 0]
    grad = torch.zeros_like(w)
    for r, g in zip(x.reshape(-1, p.nu).split(2048), back.reshape(-1, p.nu).split(2048)):
        grad += torch.autograd.grad(_network64(w, r, s), w, g)[0]
    m = torch.empty(w.shape, device=DEV, dtype=torch.float32).normal_(0.0, 1e-6, generator=_rng(seed)).double()
    v = torch.full_like(w, 1e-8).detach()
    m, v = 0.9 * m + 0.1 * grad, 0.999 * v + 0.001 * grad * grad
    t = 1001
    new = w.detach() - 1e-3 * (m / (1 - 0.9 ** t)) / ((v / (1 - 0.999 ** t)).sqrt() + 1e-8)
    return {"loss": float(diff.square().mean()), "residual": residual, "gradient": grad, "weights": new, "m": m, "v": v}
