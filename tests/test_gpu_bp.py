"""Backprojection on the GPU through the C ABI, against the oracle and the reference kernel.

FP32_EXACT must be bit-identical to the reference kernel cudaFdkBP (emulated by the oracle,
and the reference's own kernel compiled for sm_100a).  FP32 (staged) must match the
reference arithmetic within rel-L2 1e-5; MIXED (FP16 views) within rel-L2 1e-3 of FP64."""
import os

import numpy as np
import pytest

import fdk_b200 as F
from oracle import oracle as O
from tests.helpers import (knife_edge_mask, max_rel, oracle_bp_f64, oracle_bp_ref32, oracle_filtered,
                           phantom_views, rel_l2, small_param)

pytestmark = pytest.mark.gpu

REF_BP = os.path.join(O.REF_DIR, "libref_gpu_bp.so")


def run_bp(precision, p, top, bot, batches, mats_batches, transpose=1, width=None, height=None):
    width = width or p.nv
    height = height or p.nu
    bp = F.BackProjectionFDK(width, height, 32, p.nx, p.ny, p.nz, F.BoxT(*top), F.BoxT(*bot), precision)
    for f, m in zip(batches, mats_batches):
        bp.BP(transpose, f, width, height, m, f.shape[0])
    vol = bp.GetVolumeData()
    n, ms = bp.stats()
    assert n == sum(f.shape[0] for f in batches) and ms > 0
    bp.close()
    return vol


def random_views(n, h, w, seed=0):
    return np.random.default_rng(seed).standard_normal((n, h, w)).astype(np.float32)


@pytest.mark.parametrize("n,nu,nv,views", [(32, 40, 36, 16), (48, 64, 64, 40), (30, 33, 31, 7)])
def test_exact_symmetric_bitwise_vs_oracle(n, nu, nv, views):
    p = small_param(n, nu, nv, views)
    mats = p.proj_matrices()
    filt = random_views(views, nu, nv, seed=n)
    top = [0, 0, 0, n, n, n // 2]
    bot = [0, 0, n - n // 2, n, n, n // 2]
    batches = [filt[i:i + 32] for i in range(0, views, 32)]
    mb = [mats[i:i + 32] for i in range(0, views, 32)]
    got = run_bp("fp32_exact", p, top, bot, batches, mb)
    want = oracle_bp_ref32(top, bot[5], n, batches, mb)
    assert np.array_equal(got, want), (np.abs(got - want).max(), np.abs(want).max())


def test_exact_subbox_and_nonsymmetric_bitwise():
    n, views = 40, 12
    p = small_param(n, 48, 44, views)
    mats = p.proj_matrices()
    filt = random_views(views, 48, 44, seed=5)
    top = [4, 6, 8, 20, 24, 10]
    bot = [4, 6, n - 1 - 8 - 10 + 1, 20, 24, 10]
    got = run_bp("fp32_exact", p, top, bot, [filt], [mats])
    assert np.array_equal(got, oracle_bp_ref32(top, bot[5], n, [filt], [mats]))
    top2 = [0, 0, 5, n, n, 17]
    got2 = run_bp("fp32_exact", p, top2, [0, 0, 0, 0, 0, 0], [filt], [mats])
    assert np.array_equal(got2, oracle_bp_ref32(top2, 0, n, [filt], [mats]))


def test_exact_untransposed_views_bitwise():
    n, views = 32, 9
    p = small_param(n, 40, 36, views)
    mats = p.proj_matrices()
    filt_t = random_views(views, 40, 36, seed=9)           # (nu rows, nv)
    filt_r = np.ascontiguousarray(filt_t.transpose(0, 2, 1))  # (nv rows, nu)
    top = [0, 0, 0, n, n, n // 2]
    bot = [0, 0, n // 2, n, n, n // 2]
    a = run_bp("fp32_exact", p, top, bot, [filt_t], [mats], 1)
    b = run_bp("fp32_exact", p, top, bot, [filt_r], [mats], 0, width=40, height=36)
    # TRANSPOSE=0 blends along u first (the frame row), TRANSPOSE=1 along v first: same
    # samples, different rounding order
    assert rel_l2(b, a) <= 1e-6


@pytest.mark.skipif(not os.path.exists(REF_BP), reason="reference GPU build absent")
@pytest.mark.parametrize("views", [32, 45])
def test_exact_bitwise_vs_reference_kernel(views):
    """Against the reference's own cudaFdkBP compiled for sm_100a (BackProjectionFDK)."""
    n = 64
    p = small_param(n, 48, 40, views)
    mats = p.proj_matrices()
    filt = random_views(views, 48, 40, seed=11)
    top = [0, 0, 0, n, n, n // 2]
    bot = [0, 0, n // 2, n, n, n // 2]
    batches = [filt[i:i + 32] for i in range(0, views, 32)]
    mb = [mats[i:i + 32] for i in range(0, views, 32)]
    ref = O.RefGPU().backproject(batches, mb, n, n, n, top, bot)
    got = run_bp("fp32_exact", p, top, bot, batches, mb)
    assert np.array_equal(got, ref)
    assert np.array_equal(ref, oracle_bp_ref32(top, bot[5], n, batches, mb))  # pins the oracle


@pytest.mark.parametrize("kernel", ["tma", "staged"])
@pytest.mark.parametrize("precision,tol", [("fp32", 1e-5), ("mixed", 1e-3)])
@pytest.mark.parametrize("n,views", [(32, 24), (64, 64), (96, 40)])
def test_fast_paths_on_phantom(precision, tol, n, views, kernel, monkeypatch):
    """Both staged kernels: the TMA-fed persistent kernel and the synchronous-staging one."""
    if kernel == "staged":
        monkeypatch.setenv("FDK_BP_KERNEL", "staged")
    p = small_param(n, n, n, views)
    mats = p.proj_matrices()
    _, proj = phantom_views(p, seed=n)
    filt = oracle_filtered(p, proj)
    top = [0, 0, 0, n, n, n // 2]
    bot = [0, 0, n // 2, n, n, n // 2]
    batches = [filt[i:i + 32] for i in range(0, views, 32)]
    mb = [mats[i:i + 32] for i in range(0, views, 32)]
    got = run_bp(precision, p, top, bot, batches, mb)
    ref32 = oracle_bp_ref32(top, bot[5], n, batches, mb)
    f64, _ = oracle_bp_f64(top, bot[5], n, filt, p.proj_matrices(np.float64))
    m = knife_edge_mask(p, top, bot[5])
    e32, e64 = rel_l2(got[m], ref32[m]), rel_l2(got[m], f64[m])
    print(f"{precision} n={n}: rel-L2 vs reference arithmetic {e32:.2e}, vs FP64 {e64:.2e}, "
          f"max rel {max_rel(got, f64):.2e}")
    if precision == "fp32":
        assert e32 <= tol
    assert e64 <= tol


@pytest.mark.parametrize("kernel", ["tma", "staged"])
@pytest.mark.parametrize("precision", ["fp32", "mixed"])
@pytest.mark.parametrize("nu,nv", [(24, 20), (26, 21)])  # nv=21: rows not 16-byte multiples
def test_fast_border_views(precision, kernel, nu, nv, monkeypatch):
    """Detector smaller than the volume's shadow: boundary samples follow SUBPIXEL's rule."""
    if kernel == "staged":
        monkeypatch.setenv("FDK_BP_KERNEL", "staged")
    n, views = 32, 16
    p = small_param(n, nu, nv, views)  # detector crops the volume in u and v
    p.du = p.dv = 384.0 / 40
    mats = p.proj_matrices()
    filt = random_views(views, nu, nv, seed=21)
    top = [0, 0, 0, n, n, n // 2]
    bot = [0, 0, n // 2, n, n, n // 2]
    got = run_bp(precision, p, top, bot, [filt], [mats])
    want = oracle_bp_ref32(top, bot[5], n, [filt], [mats])
    m = knife_edge_mask(p, top, bot[5])
    e = rel_l2(got[m], want[m])
    print(precision, kernel, nu, nv, "rel-L2 vs reference arithmetic", e)
    # MIXED on white-noise views: FP16 samples and the 1/1024-pixel fixed-point fraction of the
    # staged gather bound the per-sample error at a few 1e-4 of the sample differences; the
    # north-star bar of 1e-3 holds even here, where neighbouring samples are uncorrelated
    assert e <= (1e-5 if precision == "fp32" else 1e-3), e


@pytest.mark.parametrize("half", [176, 190, 193])  # 1100, 1200 and 1300 tiles of 16 slices; ragged in both heights
def test_fp32_tile_heights(half):
    """FP32 tiles of 12 and of 16 slices, against FP32_EXACT.  A detector coordinate is off by at most four roundings
    of the detector's size; a sample of white noise moves by 2.2 of its own size per pixel (rms)."""
    n, nu, nv, views = 160, 40, 44, 5
    p = small_param(n, nu, nv, views)
    p.nz = 2 * half
    top, bot = [0, 0, 0, n, n, half], [0, 0, half, n, n, half]
    filt, mats = random_views(views, nu, nv, seed=half), p.proj_matrices()
    got, want = (run_bp(k, p, top, bot, [filt], [mats]) for k in ("fp32", "fp32_exact"))
    m = knife_edge_mask(p, top, bot[5])
    assert rel_l2(got[m], want[m]) <= 4 * 2.0 ** -24 * nv * 2.2


def test_fast_rejects_non_circular_matrices():
    n = 16
    p = small_param(n, 16, 16, 4)
    mats = p.proj_matrices().copy()
    mats[:, 2] = 0.01
    bp = F.BackProjectionFDK(16, 16, 32, n, n, n, F.BoxT(0, 0, 0, n, n, 8), F.BoxT(0, 0, 8, n, n, 8), "fp32")
    with pytest.raises(F.FdkError):
        bp.BP(1, random_views(4, 16, 16), 16, 16, mats, 4)


def test_exact_views_of_4_gb():
    """A view of more than 2^30 samples is addressed with 64-bit offsets: the same bits as a crop of it.  The matrix
    has w = 1 and dyadic u and v, so that moving the detector's origin by whole rows changes no rounding."""
    import torch

    n, width, rows, crop = 24, 32768, 32800, 256
    tail = random_views(1, crop, width, seed=3)
    big = torch.zeros((1, rows, width), device="cuda")
    big[:, rows - crop:] = torch.from_numpy(tail).cuda()
    small = torch.from_numpy(tail).cuda()

    def run(views, height, u0):
        m = np.array([[2.0, 0.25, 0, u0, 0.5, 16.0, 64.25, 100.5, 0, 0, 0, 1.0]], np.float32)
        bp = F.BackProjectionFDK(width, height, 1, n, n, n, F.BoxT(0, 0, 0, n, n, n), F.BoxT(0, 0, 0, 0, 0, 0))
        bp.BP_device(views.data_ptr(), F.LAYOUT_TRANSPOSED, m, 1)
        vol = bp.GetVolumeData().copy()
        bp.close()
        return vol

    got, want = run(big, rows, rows - crop + 130.5), run(small, crop, 130.5)
    assert np.array_equal(got, want) and np.abs(want).max() > 0


@pytest.mark.parametrize("nu", [64, 320, 400, 704])
def test_fp32_footprints_that_miss_the_box(nu):
    """Detectors of 0.4 to 4.4 rows a slice: all, some and none of the tiles fit the staged kernel's box, in a slab
    that fills the taller tiles better (10 x 10 columns of tiles, 216 slices: five waves of two CTAs per SM against
    seven).  The second scan of the handle has pixels of twice the size, so that its tiles are chosen anew.  Against FP32_EXACT; tolerance as
    test_fp32_tile_heights."""
    n, half, views = 160, 216, 3
    p = small_param(n, nu, nu, views)
    p.nz = 2 * half
    top, bot = [0, 0, 0, n, n, half], [0, 0, half, n, n, half]
    filt = random_views(views, nu, nu, seed=nu)
    bps = [F.BackProjectionFDK(nu, nu, 4, n, n, 2 * half, F.BoxT(*top), F.BoxT(*bot), k) for k in ("fp32", "fp32_exact")]
    for pitch in (384.0 / nu, 768.0 / nu):
        p.du = p.dv = pitch
        vols = []
        for bp in bps:
            bp.reset()
            bp.BP(1, filt, nu, nu, p.proj_matrices(), views)
            vols.append(bp.GetVolumeData().copy())
        m = knife_edge_mask(p, top, half)
        assert np.abs(vols[1]).max() > 0 and m.mean() > 0.5
        assert rel_l2(vols[0][m], vols[1][m]) <= 4 * 2.0 ** -24 * nu * 2.2
    for bp in bps:
        bp.close()


@pytest.mark.parametrize("precision,layout", [("fp32_exact", "transposed"), ("fp32_exact", "rows"), ("fp32", "mirror")])
def test_detectors_of_more_than_2_23_rows(precision, layout):
    """Detector rows beyond 2^23, where adding 2^23 no longer leaves a coordinate's whole part in the low bits, against
    a crop of the detector.  w = 1, u dyadic and v whole, so that moving the origin changes no rounding: FP32_EXACT gives
    the same bits, FP32, which takes another kernel, three roundings of a sample.  (Top slices only: the mirror
    ones fall outside the crop.)"""
    import torch

    n, nu, rows, crop = 16, 8, (1 << 23) + 512, 512
    tail = torch.from_numpy(random_views(1, nu, crop, seed=8)).cuda()

    def run(nv, v0):
        x = torch.zeros((1, nu, nv), device="cuda")  # (views, u, v)
        x[:, :, nv - crop:] = tail
        if layout == "rows":
            x = x.transpose(1, 2).contiguous()
        if layout == "mirror":
            x = torch.stack([x, x.flip(2)], -1).contiguous()
        m = np.array([[0.25, 0, 0, 1.5, 2.0, 1.0, 8.0, v0, 0, 0, 0, 1.0]], np.float32)
        half = n // 2
        top, bot = F.BoxT(0, 0, 0, n, n, half), F.BoxT(0, 0, half, n, n, half)
        w, h = (nu, nv) if layout == "rows" else (nv, nu)
        bp = F.BackProjectionFDK(w, h, 1, n, n, n, top, bot, precision)
        if layout == "rows":
            bp.BP(0, x.cpu().numpy(), w, h, m, 1)
        else:
            bp.BP_device(x.data_ptr(), F.LAYOUT_MIRROR if layout == "mirror" else F.LAYOUT_TRANSPOSED, m, 1)
        vol = np.asarray(bp.GetVolumeData()).reshape(n, n, n)[:half].copy()
        bp.close()
        return vol

    got, want = run(rows, rows - 300.0), run(crop, crop - 300.0)
    assert np.abs(want).max() > 0
    assert np.array_equal(got, want) if precision == "fp32_exact" else max_rel(got, want) <= 2.0 ** -22


def test_adjoint_of_more_than_2_23_rows():
    """As above, the adjoint: gradient rows of the big detector and of its crop."""
    import ctypes as C

    import torch

    from fdk_b200._lib import check, lib

    n, nu, rows, crop = 16, 8, (1 << 23) + 512, 512
    res = torch.randn((n, n, n), device="cuda")
    res[n // 2:] = 0  # no mirror slices

    def run(nv):
        p = small_param(n, nu, nv, 1)
        m = torch.tensor([0.25, 0, 0, 1.5, 2.0, 1.0, 8.0, nv - 300.0, 0, 0, 0, 1.0], device="cuda")
        g = torch.zeros((1, nv, nu), device="cuda")
        check(lib().fdk_bp_adjoint(C.byref(p.to_c()), res.data_ptr(), m.data_ptr(), 1, g.data_ptr(), None))
        return g[0, nv - crop:].cpu().numpy()

    got, want = run(rows), run(crop)
    assert np.abs(got - want).max() <= 2.0 ** -16 * np.abs(want).max() and np.abs(want).max() > 0
