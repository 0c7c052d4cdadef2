"""The kernels' own FP64 square root and rotation (bp_common.cuh): built for the
host with perturbed estimates in place of the hardware's, and on the GPU beside
CUDA's sqrt."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CUDA_HOME = os.environ.get("CUDA_HOME", "/usr/local/cuda")
TWO_PI = 2 * np.longdouble("3.14159265358979323846264338327950288")


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("fp64") / "libtile_probe.so")
    subprocess.run(["g++", "-O2", "-march=native", "-std=c++20", "-ffp-contract=off", "-fPIC", "-shared", "-w", "-pthread",
                    f"-I{CUDA_HOME}/include", "-o", so, os.path.join(HERE, "native", "tile_probe.cpp")], check=True)
    return ctypes.CDLL(so)


def roots(n, seed):
    """Arguments of every size a squared range has and far beyond, exact
    squares, their neighbours and halfway cases of the mantissa."""
    rng = np.random.default_rng(seed)
    m = rng.uniform(1.0, 4.0, n) * 2.0 ** rng.integers(-400, 400, n)
    r = np.ldexp(rng.integers(1 << 26, 1 << 27, n // 8).astype(np.float64), rng.integers(-200, 200, n // 8))
    sq = (r * r)[np.isfinite(r * r)]
    edges = np.array([1.0, 2.0, 4.0, np.nextafter(1.0, 0.0), np.nextafter(1.0, 2.0), np.nextafter(4.0, 0.0), 1e-290, 1e290])
    return np.concatenate([m, sq, np.nextafter(sq, 0.0), np.nextafter(sq, np.inf), rng.uniform(1e-2, 1e14, n), edges])


def check_roots(got, x):
    """Within one unit, and the neighbour for no more than 16 of some 2.4 n
    arguments: 2^-78 before the last rounding misses a tie once in 2^24 or so."""
    want = np.sqrt(x)
    assert (np.abs(got - want) <= np.spacing(want)).all()
    assert np.count_nonzero(got != want) <= 16, np.count_nonzero(got != want)


def phases(n, seed):
    rng = np.random.default_rng(seed)
    edges = np.arange(-64, 65) / 8.0
    return np.concatenate([rng.uniform(-s, s, n) for s in (1.0, 1e3, 1e6, 1e12, 2.0 ** 49)] +
                          [edges, np.nextafter(edges, 9.0), np.nextafter(edges, -9.0), [2.0 ** 49, -(2.0 ** 49), 0.0]])


def check_turns(cs, sn, ph):
    """Two roundings of the sine's polynomial and product, one of the cosine's
    and a small part of another: 3e-16."""
    exact = TWO_PI * (ph - np.rint(ph)).astype(np.longdouble)
    assert np.abs(cs - np.cos(exact)).max() < 3e-16
    assert np.abs(sn - np.sin(exact)).max() < 3e-16


def test_square_root_from_perturbed_estimates(host):
    x = roots(1 << 21, 1)
    out = np.empty_like(x)
    host.sqrt_probe(x.ctypes.data_as(ctypes.c_void_p), out.ctypes.data_as(ctypes.c_void_p), ctypes.c_int(len(x)))
    check_roots(out, x)


def test_rotation(host):
    ph = phases(200000, 2)
    cs, sn = np.empty_like(ph), np.empty_like(ph)
    host.rotation_probe(*(v.ctypes.data_as(ctypes.c_void_p) for v in (ph, cs, sn)), ctypes.c_int(len(ph)))
    check_turns(cs, sn, ph)


@pytest.mark.gpu
def test_on_the_gpu():
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from uncc_sar_focusing_b200 import build as B

    lib = ctypes.CDLL(B.PROBE_LIB)
    lib.sarbp_probe_math.argtypes = [ctypes.c_int, ctypes.c_void_p, ctypes.c_void_p, ctypes.c_void_p, ctypes.c_int]
    for which, x in ((0, roots(1 << 22, 3)), (1, phases(200000, 4))):
        d = torch.as_tensor(x).cuda()
        a, b = torch.empty_like(d), torch.empty_like(d)
        torch.cuda.synchronize()
        assert lib.sarbp_probe_math(which, d.data_ptr(), a.data_ptr(), b.data_ptr(), len(x)) == 0
        a, b = a.cpu().numpy(), b.cpu().numpy()
        if which == 0:
            check_roots(a, x)
            assert (b == np.sqrt(x)).all()
        else:
            check_turns(a, b, x)
