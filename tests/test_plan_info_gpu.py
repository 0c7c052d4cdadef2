"""The launches a plan says it makes (sarbp_plan_get_info) against those it
makes, counted by the CUDA profiler's activity records."""
import numpy as np
import pytest

from uncc_sar_focusing_b200 import scenes as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,pregeo", [("mixed", True), ("mixed", False), ("fp64", True)])
def test_launches_of_a_focus_call(monkeypatch, precision, pregeo):
    import torch
    from torch.profiler import ProfilerActivity, profile

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from uncc_sar_focusing_b200 import focusing

    if not pregeo:
        monkeypatch.setenv("SARBP_PREGEO", "0")
    sc = S.point_target_scene(K=256, Np=40, n=70, spacing=0.1, nfft=1024, snr_db=None, seed=3, n_targets=2)
    dev = [torch.as_tensor(np.ascontiguousarray(a)).cuda()
           for a in (sc.phase_history, sc.ant_x, sc.ant_y, sc.ant_z, sc.slant_range, sc.start_freq)]
    with focusing.Plan.for_scene(sc, precision) as plan:
        info = plan.info
        out = plan.new_image("cuda")
        plan.focus(*dev, out=out)
        torch.cuda.synchronize()
        with profile(activities=[ProfilerActivity.CUDA]) as prof:
            plan.focus(*dev, out=out)
            torch.cuda.synchronize()
    names = [e.name for e in prof.events() if "sarbp" in e.name or "bp_" in e.name or "rc_" in e.name]
    assert info["geometry_record_kernels"] == int(precision == "mixed" and pregeo)
    if not prof.events():
        pytest.skip("the profiler records no activity here")
    assert sum("geo_records" in n for n in names) == info["geometry_record_kernels"]
    ours = [n for n in names if "rc_" in n or "bp_" in n]
    assert len(ours) == 1 + info["geometry_record_kernels"] + info["kernels_per_backproject"], names
