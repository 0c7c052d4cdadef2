"""The mixed kernels' per-(tile, pulse) arithmetic from its own source, on the CPU.

native/tile_probe.cpp builds csrc/bp_tile.cuh for the host: records, polynomial
tables and every thread's phases and bins of one tile, against the exact range
in FP64.  A bin becomes a shared-memory address in the kernels, so each must be
finite and inside the pulse's window whatever the start frequency is.
"""
import ctypes
import math
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CUDA_HOME = os.environ.get("CUDA_HOME", "/usr/local/cuda")
C = 299792458.0
PG_NEAR = 4


@pytest.fixture(scope="module")
def probe(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("tile_probe") / "libtile_probe.so")
    subprocess.run(["g++", "-O2", "-std=c++20", "-ffp-contract=off", "-fPIC", "-shared", "-w", "-pthread",
                    f"-I{CUDA_HOME}/include", "-o", so, os.path.join(HERE, "native", "tile_probe.cpp")], check=True)
    lib = ctypes.CDLL(so)
    d, i, p = ctypes.c_double, ctypes.c_int, ctypes.c_void_p
    lib.tile_probe.argtypes = [p, i, i, d, d, d, d, d, i, d, d, i, i, i, p, p, p]
    return lib.tile_probe


def tile(probe, f0, radius, spacing, mx, exchanged=False, split=False, nfft=3392, lam=32.1, el=30.0,
         look=(0.0, 30.0, 88.0, 200.0), near=1.0, origin=(0.3, -0.7)):
    """The tile's phases, bins and pulse words, with their exact values:
    phase modulo one turn, window-centred bin (float64).  near: a factor on the
    far-field test's constant."""
    az = np.radians(np.asarray(look))
    n = len(az)
    x = radius * math.cos(math.radians(el)) * np.cos(az)
    y = radius * math.cos(math.radians(el)) * np.sin(az)
    z = np.full(n, radius * math.sin(math.radians(el)))
    r0 = np.sqrt(x * x + y * y + z * z)
    f = np.broadcast_to(np.asarray(f0, dtype=np.float64), (n,))
    geo = np.ascontiguousarray(np.stack([x, y, z, r0, f]))
    dx, dy = spacing, 1.1 * spacing
    left, bottom = origin
    hd = math.hypot(4 * mx * dx, 32 * dy)
    W = int(math.ceil(lam * hd)) + 3
    P = np.full((n, 8 * mx, 64), np.nan, dtype=np.float32)
    B = P.copy()
    words = np.zeros((n, 3), dtype=np.int32)
    err = probe(geo.ctypes.data, n, nfft, lam, dx, dy, left, bottom, W, 16.0 * hd, near * 0.625 * hd ** 4 / 1e-7, mx,
                int(exchanged), int(split), P.ctypes.data, B.ctypes.data, words.ctypes.data)
    assert err == 0
    if exchanged:  # the map's rows run along the image's columns
        P, B = P.transpose(0, 2, 1), B.transpose(0, 2, 1)
    px = left + dx * np.arange(8 * mx)[None, :, None]
    py = bottom + dy * np.arange(64)[None, None, :]
    R = np.sqrt((x[:, None, None] - px) ** 2 + (y[:, None, None] - py) ** 2 + z[:, None, None] ** 2)
    dR = R - r0[:, None, None]
    rev = 2.0 * f[:, None, None] / C * dR
    bin_ = lam * dR + 0.5 * nfft - words[:, 1, None, None] - W
    rc = np.sqrt((x - left - 4 * mx * dx) ** 2 + (y - bottom - 32 * dy) ** 2 + z * z)
    far = (0.625 * hd ** 4 / rc ** 3)[:, None, None]  # metres the expansion may be off
    v = np.stack([x - left - 4 * mx * dx, y - bottom - 32 * dy, z], 1)
    return dict(rc=rc, r0=r0, v=v, P=P, B=B, words=words, rev=rev, bin=bin_, far=far, kr=4.0 * math.pi * f[:, None, None] / C, lam=lam, W=W)


def check(t):
    assert np.isfinite(t["P"]).all() and np.isfinite(t["B"]).all()
    wp = t["words"][:, 2, None, None]
    fl = np.floor(t["B"])
    assert (fl >= -wp).all() and (fl <= wp).all(), "a bin outside its pulse's window"
    far = np.where(t["words"][:, 0, None, None] & PG_NEAR, 0.0, t["far"])
    # bins: four roundings at the window's half-width; phases: five at the
    # largest phase and 1e-6 rad for the cubic term's fit; and the expansion
    tol_bin = 4.0 * 2.0 ** -24 * t["W"] + t["lam"] * far
    tol_phase = 5.0 * 2.0 ** -24 * np.abs(t["P"]).max() + 1e-6 + np.abs(t["kr"]) * far
    assert (np.abs(t["B"] - t["bin"]) <= tol_bin).all(), np.abs(t["B"] - t["bin"]).max()
    turn = t["P"].astype(np.float64) / (2.0 * math.pi) - t["rev"]
    off = 2.0 * math.pi * np.abs(turn - np.rint(turn))
    assert (off <= tol_phase).all(), off.max()


@pytest.mark.parametrize("mx,exchanged", [(1, False), (2, False), (4, False), (8, False), (8, True)])
@pytest.mark.parametrize("split", [False, True])
@pytest.mark.parametrize("radius,spacing", [(8e3, 0.1), (10e3, 0.08), (60.0, 0.1), (3e3, 0.4)])
def test_phases_and_bins(probe, mx, exchanged, split, radius, spacing):
    check(tile(probe, 9.28e9, radius, spacing, mx, exchanged, split))


@pytest.mark.parametrize("radius,spacing,el,mx", [(8e3, 0.3, 45.0, 8), (8e3, 2.0, 30.0, 4), (300.0, 0.2, 20.0, 8),
                                                  (30.0, 0.1, 40.0, 8), (9.0, 0.1, 60.0, 8), (5.0, 0.1, 88.0, 1)])
def test_near_field_remainder(probe, radius, spacing, el, mx):
    """The exact path from a tile's far side to an antenna above it: bins as
    elsewhere; phases at the roundings of the remainder, six at its largest
    value (offset, its square, the difference, root, step and product) beside
    those of the linear part."""
    t = tile(probe, 9.28e9, radius, spacing, mx, el=el)
    assert (t["words"][:, 0] & PG_NEAR).all()
    assert np.isfinite(t["P"]).all() and np.isfinite(t["B"]).all()
    tol_bin = 4.0 * 2.0 ** -24 * t["W"]
    assert (np.abs(t["B"] - t["bin"]) <= tol_bin).all(), np.abs(t["B"] - t["bin"]).max()
    turn = t["P"].astype(np.float64) / (2.0 * math.pi) - t["rev"]
    off = 2.0 * math.pi * np.abs(turn - np.rint(turn))
    assert (off <= 2.0 ** -24 * (5.0 * 40.0 + 6.0 * np.abs(t["P"]).max())).all(), off.max()


@pytest.mark.parametrize("radius,spacing", [(8e3, 0.1), (60.0, 0.1)])
@pytest.mark.parametrize("f0", [0.0, 1e-30, -1e-30, 1e-9, 25.0, -3.0e8, -9.28e9, [9.28e9, 0.0, -3.0e8, 0.0]])
def test_any_start_frequency(probe, f0, radius, spacing):
    """Baseband data and blanked pulses: the bin does not depend on the start
    frequency, the phase is zero at zero."""
    for mx, split in ((2, False), (8, False), (8, True)):
        t = tile(probe, f0, radius, spacing, mx, split=split)
        check(t)
        assert (t["P"][np.broadcast_to(t["kr"] == 0.0, t["P"].shape)] == 0.0).all()


@pytest.mark.parametrize("lam", [1e-30, 1e-14, 1e-6])
def test_wide_swaths(probe, lam):
    """Range bins of kilometres and more: the phase does not depend on them."""
    check(tile(probe, 9.28e9, 8e3, 0.1, 8, lam=lam))


@pytest.mark.parametrize("mx,bound", [(8, 10.5), (4, 0.9), (2, 0.0)])
def test_cubic_term_of_the_row_steps(probe, mx, bound):
    """The k^3 term over a thread's rows k = -mx/2 .. mx/2 - 1 is carried by the
    lower terms: what is left of k^3 is `bound` at most, and the phase is off
    by 8 q30 kr / lambda times that.  At 20 half-diagonals (with the far-field
    test turned down to 16) it stands far above the roundings, against the
    expansion itself in FP64."""
    spacing, f0, lam = 0.1, 9.28e9, 32.1
    hd = math.hypot(4 * mx * spacing, 32 * 1.1 * spacing)
    radius, el = 20.0 * hd, math.degrees(math.acos(math.sqrt(1.0 / 3.0)))  # the largest cubic term along the rows
    t = tile(probe, f0, radius, spacing, mx, el=el, lam=lam, look=(-20.0, 0.0, 15.0, 170.0), near=0.0)
    assert not (t["words"][:, 0] & PG_NEAR).any()
    i = (np.arange(8 * mx) - 4 * mx)[None, :, None] * spacing
    j = (np.arange(64) - 32)[None, None, :] * 1.1 * spacing
    v, rc = t["v"], t["rc"][:, None, None]
    along = (v[:, 0, None, None] * i + v[:, 1, None, None] * j) / rc
    e = i * i + j * j - along * along
    rev = 2.0 * f0 / C * (rc - t["r0"][:, None, None] - along + e * (0.5 / rc + along * 0.5 / rc ** 2))
    turn = t["P"].astype(np.float64) / (2.0 * math.pi) - rev
    off = 2.0 * math.pi * np.abs(turn - np.rint(turn))
    u = np.abs(v[:, 0]) / t["rc"]
    q30 = (2.0 * math.pi * f0 / C / t["rc"] ** 2 * u * (1.0 - u * u)).max() * spacing ** 3
    assert off.max() <= 8.0 * bound * q30 + 5.0 * 2.0 ** -24 * np.abs(t["P"]).max(), (off.max(), 8.0 * bound * q30)


@pytest.mark.parametrize("f0", [0.0, 25.0, -1.0e6, -9.28e9])
@pytest.mark.parametrize("radius,spacing,lam,mx", [(4e3, 3.0, 2.0, 8), (2.5e3, 1.5, 6.0, 8), (900.0, 0.6, 20.0, 4)])
def test_far_field_test_of_any_start_frequency(probe, f0, radius, spacing, lam, mx):
    """Coarse tiles at 17 and more half-diagonals: with a start frequency of
    zero or below it the expansion is taken only where it leaves bins within
    1e-4 and phases within 1e-7 turns, as it is above."""
    t = tile(probe, f0, radius, spacing, mx, lam=lam)
    tol_bin = 4.0 * 2.0 ** -24 * t["W"] + 1e-4
    assert (np.abs(t["B"] - t["bin"]) <= tol_bin).all(), np.abs(t["B"] - t["bin"]).max()
    turn = t["P"].astype(np.float64) / (2.0 * math.pi) - t["rev"]
    off = 2.0 * math.pi * np.abs(turn - np.rint(turn))
    tol = 2.0 ** -24 * (5.0 * 40.0 + 6.0 * np.abs(t["P"]).max()) + 2.0 * math.pi * 1e-7 + 1e-6
    assert (off <= tol).all(), off.max()


@pytest.mark.parametrize("radius", [1e-21, 1e-19, 1e-12, 1e-3])
def test_one_pixel_next_to_the_antenna(probe, radius):
    """A grid of one pixel has a tile of no extent: no range is near field by
    its diagonal, and 1 / Rc^2 leaves FP32 at 1e-19 m.  (Below 1e-22 m the record
    itself is refused as not finite.)"""
    t = tile(probe, 9.28e9, radius, 0.0, 1, origin=(0.0, 0.0))
    assert np.isfinite(t["P"]).all() and (np.abs(t["B"] - t["bin"]) <= 1e-4).all()
