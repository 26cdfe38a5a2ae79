"""Ramp filter on the GPU against the FP64 oracle and the reference's cuFFT plugin."""
import os

import numpy as np
import pytest

import fdk_b200 as F
from oracle import oracle as O
from tests.helpers import max_rel, phantom_views, small_param

pytestmark = pytest.mark.gpu
REF_FLT = os.path.join(O.REF_DIR, "libref_gpu_filter.so")


@pytest.mark.parametrize("nu,nv", [(64, 64), (256, 256), (96, 50), (1536, 16), (2048, 8)])
@pytest.mark.parametrize("transpose", [False, True])
def test_filter_engine_vs_oracle(nu, nv, transpose):
    p = small_param(64, nu, nv, 4)
    rng = np.random.default_rng(nu + nv)
    src = (rng.standard_normal((nv, nu)) * 50 + 100).astype(np.float32)
    cos = p.cos_sigma
    eng = F.FilterEngine(cos, p.fft_kernel_real_f32)
    want = O.filter_view(src, p.fft_kernel_real, cos, pad_n=4, transpose=transpose)
    s = src.copy()
    dst = np.zeros((nu, nv) if transpose else (nv, nu), np.float32)
    eng.Filtering(s, dst, transpose)
    assert np.array_equal(s, src * cos)  # src is cosine-weighted in place, in FP32
    assert max_rel(dst, want) <= 2e-6, max_rel(dst, want)


@pytest.mark.parametrize("nu,nv", [(80, 64), (96, 50), (2048, 16), (300, 24)])
def test_device_layouts(nu, nv):
    """All device layouts against the FP64 oracle and each other.  nv = 64 and 16 take the grouped
    MIRROR kernel (row pairs tiled 2 or 4 at a time), nv = 50 the per-pair fallback, nv = 24 the
    grouped FP32 and fallback FP16 kernels."""
    import torch

    p = small_param(64, nu, nv, 6)
    _, proj = phantom_views(p)
    eng = F.FilterEngine(p.cos_sigma, p.fft_kernel_real_f32)
    src = torch.from_numpy(proj).cuda()
    want = np.stack([O.filter_view(v, p.fft_kernel_real, p.cos_sigma, pad_n=4, transpose=True) for v in proj])
    t = torch.empty((6, nu, nv), dtype=torch.float32, device="cuda")
    eng.run_device(src.data_ptr(), t.data_ptr(), 6, F.LAYOUT_TRANSPOSED, F.DTYPE_F32)
    m = torch.empty((6, nu, nv, 2), dtype=torch.float32, device="cuda")
    eng.run_device(src.data_ptr(), m.data_ptr(), 6, F.LAYOUT_MIRROR, F.DTYPE_F32)
    h = torch.empty((6, nu, nv, 2), dtype=torch.float16, device="cuda")
    scale = float(1.0 / p.cos_sigma.max())  # back to line-integral units, inside the FP16 range
    eng.run_device(src.data_ptr(), h.data_ptr(), 6, F.LAYOUT_MIRROR, F.DTYPE_F16, scale)
    r = torch.empty((6, nv, nu), dtype=torch.float32, device="cuda")
    eng.run_device(src.data_ptr(), r.data_ptr(), 6, F.LAYOUT_ROWS, F.DTYPE_F32)
    torch.cuda.synchronize()
    t, m, h, r = t.cpu().numpy(), m.cpu().numpy(), h.float().cpu().numpy() / scale, r.cpu().numpy()
    # FP32 FFT rounding grows with log2(W): 12 radix-2 stages each way at W = 4096
    assert max_rel(t, want) <= (2e-6 if nu <= 1024 else 3e-6)
    assert np.array_equal(r.transpose(0, 2, 1), t)
    assert np.array_equal(m[..., 0], t) and np.array_equal(m[..., 1], t[:, :, ::-1])
    assert max_rel(h[..., 0], want) <= 1e-3 and max_rel(h[..., 1], want[:, :, ::-1]) <= 1e-3


@pytest.mark.skipif(not os.path.exists(REF_FLT), reason="reference GPU build absent")
@pytest.mark.parametrize("nu,nv", [(64, 64), (512, 32), (256, 100)])
def test_cufft_plugin_api_vs_reference(nu, nv):
    """correct_image_real32 + filter_row_real32 == the reference's CorrectImage_Real32 +
    FilterRow_Real32 (cuFFT, pad 3) on the same device buffers."""
    import torch

    p = small_param(64, nu, nv, 3)
    rng = np.random.default_rng(7)
    views = torch.from_numpy((rng.standard_normal((3, nv, nu)) * 10).astype(np.float32)).cuda()
    table = torch.from_numpy(p.cos_sigma).cuda()
    H = torch.from_numpy(p.fft_kernel_real_f32).cuda()
    ref = O.RefGPU().filter(views.clone(), table, H, len(H)).cpu().numpy()
    a = views.clone()
    F.correct_image_real32(a, table, a)
    out = torch.empty_like(a)
    F.filter_row_real32(a, out, H)
    got = out.cpu().numpy()
    want = np.stack([O.filter_view(v, p.fft_kernel_real, p.cos_sigma, pad_n=3) for v in views.cpu().numpy()])
    assert max_rel(ref, want) <= 5e-6  # reference vs oracle
    assert max_rel(got, ref) <= 5e-6, max_rel(got, ref)


@pytest.mark.parametrize("nu,nv", [(512, 512), (1024, 64)])
def test_mirror_kernel_at_the_48k_shared_memory_boundary(nu, nv):
    """nu = 512 (W = 1024, four pairs at once) and nu = 1024 (W = 2048, two pairs) put the grouped
    MIRROR kernel at exactly 48 KiB of dynamic shared memory for FP16 and FP32 outputs."""
    import torch

    p = small_param(64, nu, nv, 2)
    rng = np.random.default_rng(nu)
    src = torch.from_numpy((rng.standard_normal((2, nv, nu)) * 10 + 40).astype(np.float32)).cuda()
    eng = F.FilterEngine(p.cos_sigma, p.fft_kernel_real_f32)
    t = torch.empty((2, nu, nv), dtype=torch.float32, device="cuda")
    eng.run_device(src.data_ptr(), t.data_ptr(), 2, F.LAYOUT_TRANSPOSED, F.DTYPE_F32)
    m = torch.empty((2, nu, nv, 2), dtype=torch.float32, device="cuda")
    eng.run_device(src.data_ptr(), m.data_ptr(), 2, F.LAYOUT_MIRROR, F.DTYPE_F32)
    h = torch.empty((2, nu, nv, 2), dtype=torch.float16, device="cuda")
    scale = float(1.0 / p.cos_sigma.max())
    eng.run_device(src.data_ptr(), h.data_ptr(), 2, F.LAYOUT_MIRROR, F.DTYPE_F16, scale)
    torch.cuda.synchronize()
    t, m = t.cpu().numpy(), m.cpu().numpy()
    assert np.array_equal(m[..., 0], t) and np.array_equal(m[..., 1], t[:, :, ::-1])
    hh = h.float().cpu().numpy() / scale
    assert max_rel(hh[..., 0], t) <= 1e-3


@pytest.mark.parametrize("nu", [1, 3, 6, 15, 16, 31, 40, 64, 127, 128, 255, 256, 511, 600, 1023, 1100, 2047, 2048])
@pytest.mark.parametrize("nv,views", [(1, 1), (7, 3), (37, 40)])
def test_every_length_and_group(nu, nv, views):
    """Every transform length (W = 2 .. 4096), one row (its own mirror), an odd row count, and few and many
    transforms per CTA, in every layout against the FP64 oracle.  Tolerances: those of the tests above (FP32
    transforms of up to 12 index bits each way; FP16 outputs round to 2^-11)."""
    import torch

    pad = min(4, nu)
    rng = np.random.default_rng(nu * 100 + nv)
    src = (rng.standard_normal((views, nv, nu)) + 2.0).astype(np.float32)
    cos = rng.uniform(0.9, 1.0, (nv, nu)).astype(np.float32)
    H = O.filter_design("hann", nu)
    want = np.stack([O.filter_view(v, H, cos, pad_n=pad, transpose=True) for v in src])
    eng = F.FilterEngine(cos, H.astype(np.float32), pad_edge=pad)
    d = torch.from_numpy(src).cuda()
    for layout, shape in ((F.LAYOUT_ROWS, (nv, nu)), (F.LAYOUT_TRANSPOSED, (nu, nv)), (F.LAYOUT_MIRROR, (nu, nv, 2))):
        for dtype, torch_dtype, tol in ((F.DTYPE_F32, torch.float32, 3e-6), (F.DTYPE_F16, torch.float16, 1e-3)):
            out = torch.full((views, *shape), 7.0, dtype=torch_dtype, device="cuda")
            eng.run_device(d.data_ptr(), out.data_ptr(), views, layout, dtype)
            got = out.double().cpu().numpy()
            if layout == F.LAYOUT_ROWS:
                got = got.transpose(0, 2, 1)
            if layout == F.LAYOUT_MIRROR:
                assert max_rel(got[..., 1], want[:, :, ::-1]) <= tol
                got = got[..., 0]
            assert max_rel(got, want) <= tol, (layout, dtype)


@pytest.mark.parametrize("log2w", range(2, 13))
@pytest.mark.parametrize("nv,views", [(1, 1), (7, 2), (37, 40)])
def test_row_entry_points_over_every_length(log2w, nv, views):
    """filter_row_real32 and its no-allocation form at every filter length they take (4 .. 4096), the shortest
    and the longest rows of each, against the FP64 oracle.  Tolerance: that of the tests above (FP32 transforms
    of up to 12 index bits each way)."""
    import ctypes as C

    import torch

    from fdk_b200._lib import DataRef, check, lib

    W = 1 << log2w
    for nu in (max(3, W // 2 + 1), W):
        rng = np.random.default_rng(W * 100 + nv)
        H = O.filter_design("hann", W // 2)  # W taps
        assert H.size == W
        src = torch.from_numpy((rng.standard_normal((views, nv, nu)) + 2.0).astype(np.float32)).cuda()
        filt = torch.from_numpy(H.astype(np.float32)).cuda()
        want = np.stack([O.filter_view(v, H, None, pad_n=3) for v in src.cpu().numpy()])
        out = torch.full_like(src, 7.0)
        F.filter_row_real32(src, out, filt)
        assert max_rel(out.cpu().numpy(), want) <= 3e-6
        again = torch.full_like(src, 7.0)
        ref = [C.byref(DataRef(t.data_ptr(), t.shape[-1], nv, views, t.shape[-1])) for t in (src, again)]
        check(lib().fdk_filter_row_real32_noalloc(*ref, C.byref(DataRef(filt.data_ptr(), W, 1, 1, W))))
        assert max_rel(again.cpu().numpy(), want) <= 3e-6


@pytest.mark.parametrize("nu", [24, 100, 200, 511, 1000, 2047, 4000])
def test_points_per_thread_agree(nu):
    """Calls of growing size hold 4, 8 and 16 points a thread, in small and large CTAs: at every length and
    layout the first view comes out alike.  The butterflies are the same; only where a stage's roots are exact
    (1 and -i) may one variant add 6e-17 of a sample that another one leaves out, so 1e-7 of the largest output
    is less than two of its last bits."""
    import torch

    nv = 37
    rng = np.random.default_rng(nu)
    cos = rng.uniform(0.9, 1.0, (nv, nu)).astype(np.float32)
    eng = F.FilterEngine(cos, O.filter_design("hann", nu).astype(np.float32))
    pairs = (nv + 1) // 2 * eng.W
    counts = sorted({max(1, n // pairs) for n in (1, 1 << 17, (1 << 17) + pairs, 1 << 19, 3 << 18, (3 << 18) + pairs, 1 << 21, 3 << 20)})
    src = torch.from_numpy((rng.standard_normal((1, nv, nu)) + 2.0).astype(np.float32)).cuda().repeat(counts[-1], 1, 1)
    for layout in (F.LAYOUT_ROWS, F.LAYOUT_TRANSPOSED, F.LAYOUT_MIRROR):
        first = None
        for n in counts:
            out = torch.full((n, nv * nu * (2 if layout == F.LAYOUT_MIRROR else 1)), 7.0, device="cuda")
            eng.run_device(src.data_ptr(), out.data_ptr(), n, layout, F.DTYPE_F32)
            first = out[:1] if first is None else first
            assert float((out - first).abs().max()) <= 1e-7 * float(first.abs().max()), (layout, n)


@pytest.mark.parametrize("nu,nv,views", [(300, 37, 1), (300, 37, 40), (2000, 5, 3), (2000, 101, 16)])
@pytest.mark.parametrize("shift", [0, 1])  # dst on a pair's boundary or on a float's
def test_middle_row_of_an_odd_detector(nu, nv, views, shift):
    """The MIRROR pair of the middle row is that row twice, as the real and as the imaginary part of its transform: the
    first is what TRANSPOSED holds, bit for bit."""
    import torch

    rng = np.random.default_rng(nu + nv)
    cos = rng.uniform(0.9, 1.0, (nv, nu)).astype(np.float32)
    eng = F.FilterEngine(cos, O.filter_design("hann", nu).astype(np.float32))
    src = torch.from_numpy((rng.standard_normal((views, nv, nu)) + 2.0).astype(np.float32)).cuda()
    t = torch.empty((views, nu, nv), device="cuda")
    m = torch.empty(views * nu * nv * 2 + shift, device="cuda")[shift:]
    eng.run_device(src.data_ptr(), t.data_ptr(), views, F.LAYOUT_TRANSPOSED, F.DTYPE_F32)
    eng.run_device(src.data_ptr(), m.data_ptr(), views, F.LAYOUT_MIRROR, F.DTYPE_F32)
    assert torch.equal(m.view(views, nu, nv, 2)[..., 0], t)


RESET = """
import ctypes as C, sys
import numpy as np
sys.path.insert(0, %r)
from fdk_b200._lib import DataRef, lib
rt = C.CDLL(%r)
rng = np.random.default_rng(3)
views, H = rng.standard_normal((3, 20, 48)).astype(np.float32), rng.uniform(0, 1, 64).astype(np.float32)
def device(a):
    p = C.c_void_p()
    assert rt.cudaMalloc(C.byref(p), C.c_size_t(a.nbytes)) == 0
    assert rt.cudaMemcpy(p, a.ctypes.data_as(C.c_void_p), C.c_size_t(a.nbytes), 1) == 0
    return p
def run():
    out = np.zeros_like(views)
    s, d, h = device(views), device(out), device(H)
    ref = lambda p, w, n, m: C.byref(DataRef(p.value, w, n, m, w))
    rc = lib().fdk_filter_row_real32(ref(s, 48, 20, 3), ref(d, 48, 20, 3), ref(h, 64, 1, 1))
    assert rc == 0, lib().fdk_last_error()
    assert rt.cudaMemcpy(out.ctypes.data_as(C.c_void_p), d, C.c_size_t(out.nbytes), 2) == 0
    return out
first = run()
assert np.array_equal(run(), first) and np.abs(first).max() > 0
assert lib().fdk_scratch_trim() == 0 and np.array_equal(run(), first)
assert rt.cudaDeviceReset() == 0
assert np.array_equal(run(), first)
print("same after a reset")
"""


def test_scratch_pool_goes_with_its_context():
    """The row filter's workspace pool is given back on request and made anew after cudaDeviceReset (a process of its
    own: a reset ends every handle of the context)."""
    import subprocess
    import sys

    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", RESET % (root, "/usr/local/cuda/lib64/libcudart.so")], capture_output=True,
                       text=True, timeout=300)
    assert r.returncode == 0 and "same after a reset" in r.stdout, r.stderr[-2000:]


def test_scratch_pool_is_given_back():
    """A projection's copy of a 134 MB volume stays in the pool until fdk_scratch_trim."""
    import ctypes as C

    import torch

    from fdk_b200._lib import check, lib

    p = small_param(320, 600, 600, 2)
    vol, out = torch.zeros((320, 320, 320), device="cuda"), torch.empty((2, 600, 600), device="cuda")
    check(lib().fdk_scratch_trim())
    free = torch.cuda.mem_get_info()[0]
    check(lib().fdk_forward_project(C.byref(p.to_c()), vol.data_ptr(), 0, 2, out.data_ptr(), None))
    held = free - torch.cuda.mem_get_info()[0]
    check(lib().fdk_scratch_trim())
    assert 100 << 20 < held <= 256 << 20 and free - torch.cuda.mem_get_info()[0] < 8 << 20
