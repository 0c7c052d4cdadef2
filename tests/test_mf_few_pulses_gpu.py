"""Matched filter of few pulses: CTAs of 16 (FP64 8), 4 and 1 warps, by the
pulse count and whether all CTAs run at once, against the FP64 oracle at the
tolerances of the other matched-filter tests."""
import numpy as np
import pytest

from oracle import oracle as O
from uncc_sar_focusing_b200 import scenes as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(19, 23), (401, 203)])
@pytest.mark.parametrize("Np", [1, 3, 4, 5, 12, 17])
@pytest.mark.parametrize("precision,tol", [("fp64", 1e-9), ("mixed", 1e-4)])
def test_few_pulses(nx, ny, Np, precision, tol):
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from uncc_sar_focusing_b200 import focusing

    sc = S.point_target_scene(K=20, Np=Np, n=36, spacing=0.15, nfft=160, snr_db=20.0, seed=8, n_targets=3, extent=1.0)
    sc.grid = S.Grid(nx=nx, ny=ny, wx=0.01 * (nx - 1), wy=0.012 * (ny - 1), x0=0.1, y0=-0.2)
    with focusing.Plan.for_scene(sc, precision) as plan:
        got = plan.matched_filter(sc.phase_history, sc.ant_x, sc.ant_y, sc.ant_z, sc.slant_range, sc.start_freq)
    assert O.rel_l2(got, O.mf_fp64(sc)) < tol
