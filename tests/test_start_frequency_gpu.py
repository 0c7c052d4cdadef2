"""Pulses with a start frequency of zero (baseband data, blanked pulses) or
next to it, through every mixed-precision entry point, against the FP64 oracle.
"""
import ctypes

import numpy as np
import pytest

from oracle import oracle as O
from uncc_sar_focusing_b200 import _native as N
from uncc_sar_focusing_b200 import scenes as S

pytestmark = pytest.mark.gpu
MIXED_TOL = 1e-4  # relative L2 of an image
GRAD_TOL = 1e-3   # of the largest gradient component
KINDS = ["zero", "blanked", "tiny", "negative"]


@pytest.fixture(scope="module")
def F():
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from uncc_sar_focusing_b200 import focusing

    return focusing


def scene(kind, **kw):
    args = dict(K=64, Np=40, n=70, spacing=0.12, nfft=512, snr_db=20.0, seed=3, n_targets=4, extent=6.0)
    args.update(kw)
    sc = S.point_target_scene(**args)
    f = np.array(sc.start_freq, dtype=np.float64)
    if kind == "zero":
        f[:] = 0.0
    elif kind == "negative":
        f[:] = -3.0e8
    else:
        f[[5, 6, 20, -1]] = 0.0 if kind == "blanked" else 1e-30
    sc.start_freq = f
    return sc


def geometry(sc):
    return sc.ant_x, sc.ant_y, sc.ant_z, sc.slant_range, sc.start_freq


def dev(a):
    import torch

    return torch.as_tensor(np.ascontiguousarray(a)).cuda()


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("kw", [dict(), dict(radius=60.0, spacing=0.1, n=64), dict(K=32, nfft=64, spacing=0.9, n=61)])
def test_image(F, kind, kw):
    sc = scene(kind, **kw)
    with F.Plan.for_scene(sc, "mixed") as plan:
        got = plan.focus(sc.phase_history, *geometry(sc))
        checked = plan.backproject(*geometry(sc), checked=True)  # raises when a bin leaves its window
    want = O.focus_fp64(sc)
    assert O.rel_l2(got, want) < MIXED_TOL
    assert O.rel_l2(checked, want) < MIXED_TOL


def test_hypotheses(F):
    tracks = [scene(k) for k in KINDS]
    sc = tracks[0]
    with F.Plan.for_scene(sc, "mixed") as plan:
        plan.range_compress(sc.phase_history)
        got = plan.backproject_hypotheses(*(np.stack([g[i] for g in map(geometry, tracks)]) for i in range(5)))
    for t, img in zip(tracks, got):
        assert O.rel_l2(img, O.focus_fp64(t)) < MIXED_TOL


def test_batch(F):
    scs = [scene(k, n=40 + 30 * i) for i, k in enumerate(KINDS)]
    with F.Batch(scs) as batch:
        imgs = batch.new_images()
        batch.focus([tuple(dev(v) for v in (sc.phase_history, *geometry(sc))) for sc in scs], imgs)
        batch.wait()
    for sc, img in zip(scs, imgs):
        assert O.rel_l2(img.cpu().numpy(), O.focus_fp64(sc)) < MIXED_TOL


def test_noalloc(F):
    import torch

    sc = scene("blanked")
    geo = [dev(v) for v in geometry(sc)]
    with F.Plan.for_scene(sc, "mixed") as plan:
        plan.range_compress(dev(sc.phase_history))
        rc = torch.empty((sc.num_pulses, sc.nfft), dtype=torch.complex64, device="cuda")
        plan.range_profiles(out=rc)
        out = plan.new_image("cuda")
        g = N.Geometry(*(v.data_ptr() for v in geo), sc.num_pulses, N.MEMORY_DEVICE)
        st = N.lib().sarbp_backproject_noalloc(ctypes.byref(plan._desc), rc.data_ptr(), ctypes.byref(g), out.data_ptr(),
                                               0, torch.cuda.current_stream().cuda_stream)
        assert st == N.SARBP_OK
        assert O.rel_l2(out.cpu().numpy(), O.focus_fp64(sc)) < MIXED_TOL


def test_adjoint(F):
    """At a start frequency of zero the gradient is the interpolation's slope
    alone, which jumps where a bin is an integer: the scene keeps the bins of
    its blanked pulses further from one than FP32 bins are off (3e-5)."""
    sc = scene("blanked")
    g = sc.grid = S.Grid(nx=17, ny=17, wx=16 * 0.31, wy=16 * 0.31, x0=0.13, y0=0.07)
    x = g.x0 - 0.5 * g.wx + g.wx / (g.nx - 1) * np.arange(g.nx)[None, :, None]
    y = g.y0 - 0.5 * g.wy + g.wy / (g.ny - 1) * np.arange(g.ny)[None, None, :]
    at = sc.start_freq == 0.0
    R = np.sqrt((sc.ant_x[at, None, None] - x) ** 2 + (sc.ant_y[at, None, None] - y) ** 2 +
                sc.ant_z[at, None, None] ** 2)
    b = (R - sc.slant_range[at, None, None]) * sc.nfft / sc.max_wr
    assert np.abs(b - np.rint(b)).min() > 3e-5
    rng = np.random.default_rng(1)
    G = (rng.standard_normal((1, 17, 17)) + 1j * rng.standard_normal((1, 17, 17))).astype(np.complex64)
    rc = O.range_compress_fp64(sc.phase_history, sc.nfft, O.window_for(sc.window, sc.num_range_samples))
    want_a, want_r = O.bp_grad_fp64(rc, *geometry(sc), sc.max_wr, g, G.astype(np.complex128))
    with F.Plan.for_scene(sc, "mixed") as plan:
        plan.range_compress(sc.phase_history)
        got_a, got_r = plan.backproject_adjoint(*geometry(sc), G)
    for got, want in ((got_a, want_a), (got_r, want_r)):
        assert np.abs(got - want).max() < GRAD_TOL * np.abs(want).max()
        # the blanked pulses by themselves: their terms are some thirty times smaller
        assert np.abs(got[..., at] - want[..., at]).max() < GRAD_TOL * np.abs(want[..., at]).max()


@pytest.mark.parametrize("f0", [0.0, -9.3e9])
def test_coarse_image(F, f0):
    """1.5 m pixels at 2.5 km, 37 half-diagonals of a tile: the expansion would
    be off by a thousandth of a bin, and by 0.05 turns at -9.3 GHz.  (The data are
    as measured at 9.3 GHz: what counts is the operator.)"""
    sc = S.point_target_scene(K=64, Np=30, n=120, spacing=1.5, nfft=512, snr_db=20.0, seed=3, n_targets=4, extent=100.0,
                              radius=2.5e3, bw=20e6)
    sc.start_freq = np.full(sc.num_pulses, f0)
    with F.Plan.for_scene(sc, "mixed") as plan:
        got = plan.focus(sc.phase_history, *geometry(sc))
        checked = plan.backproject(*geometry(sc), checked=True)
    want = O.focus_fp64(sc)
    assert O.rel_l2(got, want) < MIXED_TOL
    assert O.rel_l2(checked, want) < MIXED_TOL
