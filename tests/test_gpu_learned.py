"""Learned residual filter: the projector against the oracle, the exact backprojection adjoint
(dot-product test), the network kernels against the CPU oracle (whose own gradients are checked by
finite differences in tests/test_nn_oracle.py), the whole gradient by finite differences, a short
training that must beat plain FDK, and the committed trained network on held-out scans."""
import ctypes as C
import os

import numpy as np
import pytest

import fdk_b200 as F
from fdk_b200 import learned as Lr
from fdk_b200._lib import check, lib
from oracle import nn_oracle as N
from oracle import oracle as O
from tests.helpers import small_param

pytestmark = pytest.mark.gpu


def test_forward_projector_vs_oracle():
    import torch

    from fdk_b200.phantom import phantom_for

    p = small_param(48, 56, 40, 6)
    ell = phantom_for(p, 4, 12)
    vol = O.ellipsoid_volume(ell, p)
    d_vol = torch.from_numpy(vol).cuda()
    out = torch.empty((6, p.nv, p.nu), dtype=torch.float32, device="cuda")
    g = p.to_c()
    check(lib().fdk_forward_project(C.byref(g), d_vol.data_ptr(), 0, 6, out.data_ptr(), None))
    torch.cuda.synchronize()
    want = np.stack([O.forward_project(vol, p, a) for a in O.view_angles(p)])
    got = out.cpu().numpy()
    assert np.linalg.norm(got - want) / np.linalg.norm(want) <= 1e-4
    if os.path.exists(os.path.join(O.REF_DIR, "libref_cpu.so")):
        # and against the reference's own 3dct ForwardProjection (3dct/3dct.cpp:430-573)
        ref = np.stack([O.RefCPU().forward_projection(vol, p, i) for i in range(6)])
        assert np.linalg.norm(got - ref) / np.linalg.norm(ref) <= 1e-4


def test_bp_adjoint_dot_product():
    """<BP(p), r> == <p, BP^T(r)> for the staged FP32 backprojection and its adjoint kernel."""
    import torch

    n, views = 40, 12
    p = small_param(n, 48, 44, views)
    rng = np.random.default_rng(0)
    rows = torch.from_numpy(rng.standard_normal((views, p.nv, p.nu)).astype(np.float32)).cuda()
    r = torch.from_numpy(rng.standard_normal((n, n, n)).astype(np.float32)).cuda()  # [z][y][x]
    mirror = torch.empty((views, p.nu, p.nv, 2), dtype=torch.float32, device="cuda")
    check(lib().fdk_rows_to_mirror(rows.data_ptr(), mirror.data_ptr(), views, p.nu, p.nv, None))
    bp = F.BackProjectionFDK(p.nv, p.nu, 32, n, n, n, F.BoxT(0, 0, 0, n, n, n // 2), F.BoxT(0, 0, n // 2, n, n, n // 2),
                             "fp32")
    mats = p.proj_matrices()
    bp.BP_device(mirror.data_ptr(), F.LAYOUT_MIRROR, mats, views)
    vol = bp.GetVolumeData()  # [z][y][x] for the full slab pair
    a = float((vol.astype(np.float64) * r.cpu().numpy().astype(np.float64)).sum())
    grad = torch.zeros_like(rows)
    d_mats = torch.from_numpy(mats.reshape(-1)).cuda()
    g = p.to_c()
    check(lib().fdk_bp_adjoint(C.byref(g), r.data_ptr(), d_mats.data_ptr(), views, grad.data_ptr(), None))
    torch.cuda.synchronize()
    b = float((rows.double() * grad.double()).sum())
    assert abs(a - b) <= 1e-4 * abs(a), (a, b)


@pytest.mark.parametrize("n,nu,nv,views", [(50, 20, 20, 9), (24, 56, 52, 12), (16, 80, 76, 5), (34, 19, 45, 17)])
def test_bp_adjoint_slices_per_row(n, nu, nv, views):
    """Several slices per detector row, several rows per slice, odd sizes, views past a multiple of 8.  A detector
    coordinate of either kernel is off by at most four roundings of the detector's size, which moves a sample of
    white noise by 2.2 of its own size per pixel (rms); the sum over the volume is held to four of its deviations."""
    import torch

    p = small_param(n, nu, nv, views)
    rng = np.random.default_rng(n)
    rows = torch.from_numpy(rng.standard_normal((views, nv, nu)).astype(np.float32)).cuda()
    r = torch.from_numpy(rng.standard_normal((n, n, n)).astype(np.float32)).cuda()
    mats = p.proj_matrices()
    top, bot = (F.BoxT(0, 0, 0, n, n, n), F.BoxT(0, 0, 0, 0, 0, 0))
    bp = F.BackProjectionFDK(nv, nu, 32, n, n, n, top, bot)
    views_t = rows.transpose(1, 2).contiguous()
    bp.BP_device(views_t.data_ptr(), F.LAYOUT_TRANSPOSED, mats, views)
    vol = bp.GetVolumeData().reshape(-1).astype(np.float64).copy()
    bp.close()
    grad = torch.zeros_like(rows)
    d_mats = torch.from_numpy(mats.reshape(-1)).cuda()
    g = p.to_c()
    check(lib().fdk_bp_adjoint(C.byref(g), r.data_ptr(), d_mats.data_ptr(), views, grad.data_ptr(), None))
    torch.cuda.synchronize()
    a = float((vol * r.cpu().numpy().reshape(-1).astype(np.float64)).sum())
    b = float((rows.double() * grad.double()).sum())
    rel = 2 * 4 * 2.0 ** -24 * max(nu, nv) * 2.2
    assert abs(a - b) <= 4 * rel * float(np.linalg.norm(vol)), (a, b)


def test_network_kernels_vs_cpu_oracle():
    import torch

    rng = np.random.default_rng(1)
    rows, L, s = 37, 64, 0.25
    params = (rng.standard_normal(N.NPARAM) * 0.2).astype(np.float32)
    x = rng.standard_normal((rows, L)).astype(np.float32) * 4
    dy = rng.standard_normal((rows, L)).astype(np.float32)
    dp, dx, ddy = (torch.from_numpy(a).cuda() for a in (params, x, dy))
    y = torch.empty_like(dx)
    g = torch.empty_like(dp)
    check(lib().fdk_nn_forward(dp.data_ptr(), dx.data_ptr(), y.data_ptr(), rows, L, s, None))
    check(lib().fdk_nn_backward(dp.data_ptr(), dx.data_ptr(), ddy.data_ptr(), g.data_ptr(), rows, L, s, None))
    torch.cuda.synchronize()
    y_ref, _ = N.forward(params, x, s, round_bf16=True)
    g_ref = N.backward(params, x, dy, s, round_bf16=True)
    assert np.abs(y.cpu().numpy() - y_ref).max() <= 2e-2 * np.abs(y_ref).max()
    rel = np.linalg.norm(g.cpu().numpy() - g_ref) / np.linalg.norm(g_ref)
    assert rel <= 2e-2, rel
    assert Lr.n_params() == N.NPARAM


def test_end_to_end_gradient_finite_difference():
    """Directional derivative of the volume MSE along the last layer (W3, b3), where the loss is
    exactly quadratic in the step, from the gradient kernels (backprojection adjoint + network
    backward) against a central difference through the forward pipeline (network + BP + MSE)."""
    import torch

    p = small_param(40, 40, 40, 24)
    pl = Lr.Pipeline(p)
    x = torch.empty((p.nProj, p.nv, p.nu), dtype=torch.float32, device="cuda")
    pl.scan(7, x)
    rng = np.random.default_rng(3)
    w0 = Lr.init_params()
    k_w3 = N.NPARAM - 32 * 9 - 1
    w0[k_w3:] = (rng.standard_normal(32 * 9 + 1) * 0.05).astype(np.float32)
    d = np.zeros_like(w0)
    d[k_w3:] = rng.standard_normal(32 * 9 + 1).astype(np.float32)

    def loss(w_host, grad=False):
        w = torch.from_numpy(w_host).cuda()
        pl.truth_of(7)
        pl.reconstruct(w, x)
        e = pl.mse(grad)
        if grad:
            pl.gradient(w, x)
            torch.cuda.synchronize()
            return e, pl.dparams.cpu().numpy().astype(np.float64)
        return e

    l0, g = loss(w0, grad=True)
    t = 0.05 * l0 / abs(float(g @ d))
    wp, wm = (w0 + t * d).astype(np.float32), (w0 - t * d).astype(np.float32)
    predicted = float(g @ (wp.astype(np.float64) - wm))
    measured = loss(wp) - loss(wm)
    assert abs(measured - predicted) <= 1e-2 * abs(predicted), (measured, predicted)


def test_short_training_beats_plain_fdk():
    """A few Adam steps on a handful of small noisy scans already lower the volume error below the
    plain Hann-ramp reconstruction of the same scans."""
    import torch

    p = small_param(48, 48, 48, 30)
    pl = Lr.Pipeline(p)
    xs = torch.empty((4, p.nProj, p.nv, p.nu), dtype=torch.float32, device="cuda")
    for i in range(4):
        pl.scan(100 + i, xs[i])
    w = torch.from_numpy(Lr.init_params()).cuda()
    m, v = torch.zeros_like(w), torch.zeros_like(w)
    plain = []
    for i in range(4):
        pl.truth_of(100 + i)
        pl.reconstruct(None, xs[i])
        plain.append(pl.mse(False))
    step = 0
    for ep in range(15):
        for i in range(4):
            pl.truth_of(100 + i)
            pl.reconstruct(w, xs[i])
            pl.mse(True)
            pl.gradient(w, xs[i])
            step += 1
            check(lib().fdk_adam_step(w.data_ptr(), pl.dparams.data_ptr(), m.data_ptr(), v.data_ptr(), w.numel(), 1e-3,
                                      0.9, 0.999, 1e-8, step, None))
    learned = []
    for i in range(4):
        pl.truth_of(100 + i)
        pl.reconstruct(w, xs[i])
        learned.append(pl.mse(False))
    assert np.mean(learned) < 0.97 * np.mean(plain), (np.mean(learned), np.mean(plain))


def test_trained_weights_beat_plain_fdk_on_held_out_scans():
    """The committed C5 network (fdk_b200/weights/residual_c5.npz) against plain Hann-ramp FDK on
    held-out phantoms (seeds outside the training range): lower volume MSE on every scan and a
    clear mean gain.  The full 200-scan evaluation is fdk_b200.train_learned's output."""
    import os

    path = os.path.join(os.path.dirname(Lr.__file__), "weights", "residual_c5.npz")
    d = np.load(path)
    window = str(d["input_window"]) if "input_window" in d.files else None
    ev = Lr.evaluate(d["params"], n_test=8, seed0=5000, input_window=window)
    print(ev)
    assert ev["learned_better_frac"] == 1.0
    assert ev["mse_reduction"] >= 0.10, ev


def test_field_of_view_weights_beat_plain_fdk_inside_the_field_of_view():
    """The C5 network trained on the loss over the fully sampled field of view
    (fdk_b200/weights/residual_c5_fov.npz, `train_learned --loss-region fov`) against plain FDK
    on held-out phantoms: lower MSE on every scan, and inside the field of view a larger cut than
    the volume-trained weights give there (the 200-scan figures are in residual_c5_fov.json)."""
    import os

    path = os.path.join(os.path.dirname(Lr.__file__), "weights", "residual_c5_fov.npz")
    d = np.load(path)
    ev = Lr.evaluate(d["params"], n_test=8, seed0=5000)
    print(ev)
    assert ev["learned_better_frac"] == 1.0
    assert ev["fov_mse_reduction"] >= 0.17, ev


@pytest.mark.parametrize("nx,ny,nz,nu,nv,views", [
    (40, 40, 40, 48, 32, 3), (33, 50, 21, 70, 33, 2), (64, 64, 64, 5, 7, 1), (17, 19, 23, 40, 1, 2),
    (30, 34, 1, 64, 65, 2), (2, 3, 64, 31, 31, 4)])
def test_forward_projector_of_a_linear_volume(nx, ny, nz, nu, nv, views):
    """A volume linear in the voxel indices is reproduced by trilinear samples, so every pixel is known in FP64:
    the sum over the ray's samples.  Odd sizes, one row, one slice, few rays.  Tolerance: FP32 positions are off by about 1e-4 of the volume's extent; a ray
    whose length is a whole number of steps to 1e-2 may take one sample more or less."""
    import torch

    p = small_param(64, nu, nv, views)
    p.nx, p.ny, p.nz = nx, ny, nz
    p.dx = p.dy = p.dz = 256.0 / max(nx, ny, nz)
    z, y, x = (torch.arange(n, device="cuda", dtype=torch.float32) for n in (nz, ny, nx))
    cx, cy, cz, c0 = 1.0 / nx, 2.0 / ny, 3.0 / nz, 1.0
    vol = (c0 + cx * x[None, None, :] + cy * y[None, :, None] + cz * z[:, None, None]).contiguous()
    out = torch.full((views, nv, nu), -1.0, device="cuda")
    g = p.to_c()
    check(lib().fdk_forward_project(C.byref(g), vol.data_ptr(), 0, views, out.data_ptr(), None))
    got = out.double().cpu().numpy()
    u = (np.arange(nu) - (nu - 1) / 2) * p.du
    v = ((nv - 1) / 2 - np.arange(nv)) * p.dv
    step = p.dx
    half = (np.array([nx, ny, nz]) - 1) / 2 * step
    for i, a in enumerate(p.angles):
        c, s = np.cos(-a), np.sin(-a)
        far = p.SID - p.SOD
        o = np.array([p.SOD * s, -p.SOD * c, 0.0])
        d = np.stack([np.broadcast_to(u * c - far * s, (nv, nu)), np.broadcast_to(u * s + far * c, (nv, nu)),
                      np.broadcast_to(v[:, None], (nv, nu))], -1) - o
        d /= np.linalg.norm(d, axis=-1, keepdims=True)
        with np.errstate(divide="ignore", invalid="ignore"):
            lo, hi = (-half - o) / d, (half - o) / d
        near, end = np.fmax.reduce(np.fmin(lo, hi), -1), np.fmin.reduce(np.fmax(lo, hi), -1)
        length = np.maximum(end - near, 0) / step
        k = np.ceil(length)
        t = near + (k - 1) / 2 * step  # the samples' mean position
        pos = [o[0] / step + (nx - 1) / 2 + d[..., 0] / step * t, (ny - 1) / 2 - (o[1] + d[..., 1] * t) / step,
               (nz - 1) / 2 - (o[2] + d[..., 2] * t) / step]
        want = np.where(k > 0, k * step * (c0 + cx * pos[0] + cy * pos[1] + cz * pos[2]), 0)
        slack = 7.0 * step * (np.abs(length - np.round(length)) < 1e-2)  # the largest voxel, one sample
        off = np.abs(got[i] - want)
        assert (off <= 2e-4 * max(np.abs(want).max(), step) + slack).all(), off.max()


@pytest.mark.parametrize("nx,ny,nz,nu,nv", [(50, 50, 50, 65, 65), (45, 60, 33, 120, 35), (1030, 1030, 1030, 2070, 2070)])
def test_forward_projector_routes_agree(nx, ny, nz, nu, nv):
    """One view here has too few rays for the reordered copy of the volume and reads the volume as it is, two
    views read the copy (through 64-bit offsets above 2^30 voxels): the same arithmetic, so the same bits."""
    import torch

    p = small_param(64, nu, nv, 2)
    p.nx, p.ny, p.nz = nx, ny, nz
    p.dx = p.dy = p.dz = 256.0 / max(nx, ny, nz)
    least = (2 if nx < 1000 else 8) * nx * ny  # rays that take the copy
    assert nu * nv < least <= 2 * nu * nv
    gen = torch.Generator(device="cuda").manual_seed(nx)
    vol = torch.rand((nz, ny, nx), device="cuda", generator=gen)
    both, one = torch.empty((2, nv, nu), device="cuda"), torch.empty((2, nv, nu), device="cuda")
    g = p.to_c()
    check(lib().fdk_forward_project(C.byref(g), vol.data_ptr(), 0, 2, both.data_ptr(), None))
    for i in range(2):
        check(lib().fdk_forward_project(C.byref(g), vol.data_ptr(), i, 1, one[i].data_ptr(), None))
    assert torch.equal(both, one)
    assert float(both.abs().max()) > 0


@pytest.mark.parametrize("L,rows", [(9, 1), (9, 61), (10, 38), (60, 9), (61, 8), (84, 7), (124, 3), (126, 5), (127, 2), (128, 3),
                                    (129, 1), (200, 2), (252, 4), (255, 3), (256, 1), (256, 300)])
@pytest.mark.parametrize("offset", [0, 1])
def test_network_kernels_over_lengths(L, rows, offset):
    """Rows that share a step of 256 positions, rows that fill one tile or two, a last step that is not full,
    more steps than CTAs, and parameters on 4-byte boundaries, against the FP64 network with the same BF16
    activations.  Tolerance 2^-8: an FP32 activation next to the middle of two BF16 values may round to the
    other one, one step of 2^-8 of it, and nothing else is above 1e-6."""
    import torch

    rng = np.random.default_rng(L * 1000 + rows)
    s = 0.25
    params = (rng.standard_normal(N.NPARAM) * 0.1).astype(np.float32)
    x = rng.standard_normal((rows, L)).astype(np.float32) * 4
    dy = rng.standard_normal((rows, L)).astype(np.float32)
    dp = torch.empty(N.NPARAM + offset, device="cuda")[offset:]
    dp.copy_(torch.from_numpy(params))
    dx, ddy = (torch.from_numpy(a).cuda() for a in (x, dy))
    y, g = torch.full_like(dx, 7.0), torch.full_like(dp, 7.0)
    check(lib().fdk_nn_forward(dp.data_ptr(), dx.data_ptr(), y.data_ptr(), rows, L, s, None))
    check(lib().fdk_nn_backward(dp.data_ptr(), dx.data_ptr(), ddy.data_ptr(), g.data_ptr(), rows, L, s, None))
    torch.cuda.synchronize()
    y_ref, _ = N.forward(params, x, s, round_bf16=True)
    g_ref = N.backward(params, x, dy, s, round_bf16=True)
    assert np.abs(y.double().cpu().numpy() - y_ref).max() <= 2.0 ** -8 * np.abs(y_ref).max()
    got = g.double().cpu().numpy()
    at = 0
    for name, n in (("W1", 288), ("b1", 32), ("W2", 9216), ("b2", 32), ("W3", 288), ("b3", 1)):
        a, b = got[at:at + n], g_ref[at:at + n]
        assert np.linalg.norm(a - b) <= 2.0 ** -8 * max(np.linalg.norm(b), 1e-3 * np.linalg.norm(g_ref)), name
        at += n


@pytest.mark.parametrize("nx,ny,nz,n_ell", [(1, 1, 1, 3), (31, 33, 5, 12), (64, 35, 40, 30), (130, 20, 66, 64), (40, 40, 40, 0)])
def test_voxelizer_vs_fp64(nx, ny, nz, n_ell):
    """Voxels against the FP64 formula in numpy, ellipsoids with voxel centres exactly on their surface, flat and
    point-like ones and an axis of 0 among them.  A voxel may only differ where q is within 1e-12 of 1 (the order
    of FP64 sums)."""
    import torch

    from fdk_b200.phantom import random_ellipsoids

    p = small_param(64, 64, 64, 4)
    p.nx, p.ny, p.nz = nx, ny, nz
    p.dx, p.dy, p.dz = 1.0, 1.25, 0.75
    e = random_ellipsoids(nx + n_ell, max(n_ell, 1), 0.5 * max(nx, ny, nz))
    if n_ell > 6:
        e[0, :3], e[0, 3:6], e[0, 6:15] = 0.0, 4.0, np.eye(3).ravel()
        e[1, 3], e[2, 3:6], e[3, 5] = 1e-3, 1e-3, 0.0
    e = np.ascontiguousarray(e[:max(n_ell, 1)])
    out = torch.full((nz, ny, nx), 9.0, device="cuda")
    check(lib().fdk_voxelize(C.byref(p.to_c()), e.ctypes.data, n_ell, out.data_ptr(), None))
    z, y, x = np.meshgrid(np.arange(nz), np.arange(ny), np.arange(nx), indexing="ij")
    P = np.stack([(x - (nx - 1) / 2) * p.dx, -(y - (ny - 1) / 2) * p.dy, -(z - (nz - 1) / 2) * p.dz], -1)
    want, close = np.zeros(P.shape[:3]), np.zeros(P.shape[:3], bool)
    for k in range(n_ell):
        with np.errstate(divide="ignore", invalid="ignore"):
            q = (((P - e[k, :3]) @ e[k, 6:15].reshape(3, 3)) ** 2 / e[k, 3:6] ** 2).sum(-1)
        want += np.where(q <= 1.0, e[k, 15], 0.0)
        close |= np.abs(q - 1) < 1e-12
    got = out.cpu().numpy()
    assert (np.abs(got - want) <= 1e-6)[~close].all() and np.isfinite(got).all()


@pytest.mark.parametrize("rows", [3, 700])  # one step a CTA, and several for the one that stalls
def test_network_wait_that_runs_out_is_reported_at_once(rows, monkeypatch):
    """FDK_BP_TEST_WITHHOLD makes CTA 0 withhold its products' commit; with a 1 ms limit it gives up.  fdk_nn_check
    reports it once, what the CTA owed is not a number, and the next calls give what they gave before."""
    import torch

    L = 200
    rng = np.random.default_rng(rows)
    dp = torch.from_numpy((rng.standard_normal(N.NPARAM) * 0.1).astype(np.float32)).cuda()
    x, dy = (torch.from_numpy(rng.standard_normal((rows, L)).astype(np.float32)).cuda() for _ in range(2))

    def run():
        y, g = torch.full_like(x, 7.0), torch.full_like(dp, 7.0)
        check(lib().fdk_nn_forward(dp.data_ptr(), x.data_ptr(), y.data_ptr(), rows, L, 0.25, None))
        rc = [lib().fdk_nn_check(None)]
        check(lib().fdk_nn_backward(dp.data_ptr(), x.data_ptr(), dy.data_ptr(), g.data_ptr(), rows, L, 0.25, None))
        return y.cpu().numpy(), g.cpu().numpy(), rc + [lib().fdk_nn_check(None), lib().fdk_nn_check(None)]

    want, grad, rc = run()
    assert rc == [0, 0, 0] and np.isfinite(want).all() and np.isfinite(grad).all()
    monkeypatch.setenv("FDK_BP_WAIT_NS", "1000000")
    monkeypatch.setenv("FDK_BP_TEST_WITHHOLD", "1")
    y, g, rc = run()
    assert rc == [-7, -7, 0]  # FDK_ERR_DEVICE_CHECK, once each
    gone = np.isnan(y).all(1)
    assert gone[0] and not gone.all() and (rows == 3) == (gone.sum() == 1)
    assert np.array_equal(y[~gone], want[~gone]) and np.isnan(g).all()
    monkeypatch.delenv("FDK_BP_WAIT_NS")
    monkeypatch.delenv("FDK_BP_TEST_WITHHOLD")
    y, g, rc = run()
    assert rc == [0, 0, 0] and np.array_equal(y, want)
    assert np.abs(g - grad).max() <= 1e-5 * np.abs(grad).max()  # the order of the CTAs' FP32 additions


def test_voxelizer_keeps_points():
    """Ellipsoids far smaller than a voxel, each centred on one, turned at random: that voxel is inside (q = 0 in FP64),
    however large FP32's error of l / a is."""
    import torch

    p = small_param(64, 64, 64, 4)
    p.dx = p.dy = p.dz = 1.0
    rng = np.random.default_rng(4)
    e = np.zeros((64, 16))
    at = rng.permutation(64 ** 3)[:64]
    z, y, x = np.unravel_index(at, (64, 64, 64))
    e[:, :3] = np.stack([x - 31.5, 31.5 - y, 31.5 - z], -1)
    e[:, 3:6] = 10.0 ** rng.uniform(-9, -4, (64, 3))
    e[:, 6:15] = [np.linalg.qr(rng.standard_normal((3, 3)))[0].ravel() for _ in range(64)]
    e[:, 15] = 1.0
    out = torch.full((64, 64, 64), 9.0, device="cuda")
    check(lib().fdk_voxelize(C.byref(p.to_c()), e.ctypes.data, 64, out.data_ptr(), None))
    want = np.zeros(64 ** 3, np.float32)
    want[at] = 1.0
    assert np.array_equal(out.cpu().numpy().ravel(), want)


def test_voxelizer_of_a_long_line():
    """2,200,000 rows of one voxel: more 32-row tiles than a grid's second and third dimensions take."""
    import torch

    p = small_param(64, 64, 64, 4)
    p.nx, p.ny, p.nz = 1, 2200000, 1
    p.dx = p.dy = p.dz = 1.0
    e = np.zeros((1, 16))
    e[0, 1], e[0, 3:6], e[0, 6:15], e[0, 15] = -1e6, 100.25, np.eye(3).ravel(), 1.0
    out = torch.full((p.ny,), 9.0, device="cuda")
    check(lib().fdk_voxelize(C.byref(p.to_c()), e.ctypes.data, 1, out.data_ptr(), None))
    y = -(torch.arange(p.ny, device="cuda", dtype=torch.float64) - (p.ny - 1) / 2)
    assert torch.equal(out, ((y + 1e6).abs() <= 100.25).float())


@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
@pytest.mark.parametrize("nu", [24, 128])  # footprints that fit a tile's box, and eight times finer pixels, whose do not
def test_adjoint_of_residuals_that_are_not_finite(bad, nu):
    """The pixels of a residual that is not finite are not finite either, all others keep their values."""
    import torch

    n = 16
    p = small_param(n, nu, nu, 3)
    rng = np.random.default_rng(2)
    res = torch.from_numpy(rng.standard_normal((n, n, n)).astype(np.float32)).cuda()
    mats = p.proj_matrices().reshape(-1, 12)
    d_mats = torch.from_numpy(mats.reshape(-1)).cuda()
    z, y, x = 3, 5, 9

    def adjoint(r):
        g = torch.zeros((3, nu, nu), device="cuda")
        check(lib().fdk_bp_adjoint(C.byref(p.to_c()), r.data_ptr(), d_mats.data_ptr(), 3, g.data_ptr(), None))
        return g.cpu().numpy()

    one = torch.zeros_like(res)
    one[z, y, x] = 1.0
    touched = adjoint(one) != 0
    assert touched.sum() == 12
    want = adjoint(res)
    res[z, y, x] = bad
    got = adjoint(res)
    assert not np.isfinite(got[touched]).any()
    # a tile adds in fixed point (2^-19 of its largest term) where its residuals are finite, in FP32 where not
    assert np.abs(got - want)[~touched].max() <= 2.0 ** -16 * np.abs(want).max()
