"""Range-bin windows so wide that a stage holds one pulse, on two CTAs an SM
and on one: image and gradient against the FP64 oracle at the tolerances of the
other parity tests (images 1e-4 relative L2, gradients 1e-3 of the largest)."""
import numpy as np
import pytest

from oracle import oracle as O
from uncc_sar_focusing_b200 import scenes as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("spacing,radius,one_cta", [(0.036, 10e3, False), (0.075, 10e3, True), (0.075, 200.0, True),
                                                    (0.06, 10e3, True)])
def test_one_pulse_stages(spacing, radius, one_cta):
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from uncc_sar_focusing_b200 import focusing

    sc = S.point_target_scene(K=64, Np=21, n=40, spacing=spacing, nfft=16384, snr_db=20.0, seed=5, n_targets=3,
                              extent=20 * spacing, radius=radius)
    sc.grid = S.Grid(nx=13, ny=70, wx=12 * spacing, wy=69 * spacing, x0=0.1, y0=-0.05)
    geo = (sc.ant_x, sc.ant_y, sc.ant_z, sc.slant_range, sc.start_freq)
    rng = np.random.default_rng(3)
    G = (rng.standard_normal((1, 13, 70)) + 1j * rng.standard_normal((1, 13, 70))).astype(np.complex64)
    rc = O.range_compress_fp64(sc.phase_history, sc.nfft, O.window_for(sc.window, sc.num_range_samples))
    want_a, want_r = O.bp_grad_fp64(rc, *geo, sc.max_wr, sc.grid, G.astype(np.complex128))
    with focusing.Plan.for_scene(sc, "mixed") as plan:
        assert plan.info["stage_pulses"] == 1 and (plan.info["smem_bytes"] > 113 * 1024) == one_cta
        img = plan.focus(sc.phase_history, *geo)
        checked = plan.backproject(*geo, checked=True)
        got_a, got_r = plan.backproject_adjoint(*geo, G)
    want = O.focus_fp64(sc)
    assert O.rel_l2(img, want) < 1e-4 and O.rel_l2(checked, want) < 1e-4
    scale = max(np.abs(want_a).max(), np.abs(want_r).max())
    assert np.abs(got_a - want_a).max() < 1e-3 * scale and np.abs(got_r - want_r).max() < 1e-3 * scale
