"""Tile windows of any swath and spacing (host_common.h, built for the host): a
window wider than the kernels hold is told as one, never wrapped to a small
one that the copies and gathers would run past."""
import ctypes
import math
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CUDA_HOME = os.environ.get("CUDA_HOME", "/usr/local/cuda")
LIMIT = 1 << 16  # entries; wider windows are refused


@pytest.fixture(scope="module")
def window(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("window_probe") / "libwindow_probe.so")
    subprocess.run(["g++", "-O2", "-std=c++20", "-fPIC", "-shared", "-w", f"-I{CUDA_HOME}/include", "-o", so,
                    os.path.join(HERE, "native", "window_probe.cpp")], check=True)
    lib = ctypes.CDLL(so)

    def call(lam, dx, dy, mx):
        W, wsize = ctypes.c_int(), ctypes.c_int()
        lib.window_probe(ctypes.c_double(lam), ctypes.c_double(dx), ctypes.c_double(dy), mx, ctypes.byref(W),
                         ctypes.byref(wsize))
        return W.value, wsize.value

    return call


@pytest.mark.parametrize("mx", [1, 8])
@pytest.mark.parametrize("lam", [1e-3, 32.0, 1e4, 1e6, 1e10, 1e30, 1e300, math.inf])
def test_windows_hold_the_tile_or_are_refused(window, lam, mx):
    for spacing in (0.0, 0.01, 0.1, 10.0):
        W, wsize = window(lam, spacing, spacing, mx)
        hd = math.hypot(4 * mx * spacing, 32 * spacing)
        need = lam * hd  # bins each side; not a number where an infinite scale meets one pixel
        assert wsize == 2 * W + 2 and wsize > 0
        assert wsize > LIMIT or W >= need + 3, (W, wsize, need)


@pytest.mark.gpu
def test_plans_and_batches_refuse_them():
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from uncc_sar_focusing_b200 import _native as N
    from uncc_sar_focusing_b200 import focusing
    from uncc_sar_focusing_b200 import scenes as S

    grid = S.Grid(nx=64, ny=64, wx=6.3, wy=6.3)
    for precision in ("mixed", "fp64"):
        with pytest.raises(N.SarbpError) as e:
            focusing.Plan(64, 8, 512, 1e-8, grid, precision=precision)
        assert e.value.status == N.SARBP_ERR_UNSUPPORTED
    d = N.PlanDesc()
    d.num_range_samples, d.num_pulses, d.nfft, d.max_wr = 64, 8, 512, 1e-8
    d.grid = N.Grid(64, 64, 1, 0.0, 0.0, 0.0, 6.3, 6.3, 0.0)
    d.device = -1
    h = ctypes.c_void_p()
    assert N.lib().sarbp_batch_create(ctypes.byref(d), 1, ctypes.byref(h)) == N.SARBP_ERR_UNSUPPORTED
    x = torch.zeros(8 * 512, dtype=torch.complex64, device="cuda")
    g = torch.ones((5, 8), dtype=torch.float64, device="cuda")
    geo = N.Geometry(*(g[i].data_ptr() for i in range(5)), 8, N.MEMORY_DEVICE)
    img = torch.zeros(64 * 64, dtype=torch.complex64, device="cuda")
    st = N.lib().sarbp_backproject_noalloc(ctypes.byref(d), x.data_ptr(), ctypes.byref(geo), img.data_ptr(), 0,
                                           torch.cuda.current_stream().cuda_stream)
    assert st == N.SARBP_ERR_UNSUPPORTED
