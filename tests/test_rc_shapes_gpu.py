"""Every fused range-compression shape against the FP64 oracle, at the
tolerance of the other paths: one pulse, and a few (each CTA's next pulse is
loaded ahead, so the last one has none)."""
import numpy as np
import pytest

from oracle import oracle as O
from uncc_sar_focusing_b200 import scenes as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K", [256, 512, 1024])
@pytest.mark.parametrize("R", [1, 2, 4, 8, 16])
def test_direct_shapes(K, R):
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from uncc_sar_focusing_b200 import focusing

    sc = S.point_target_scene(K=K, Np=5, n=16, spacing=0.2, nfft=R * K, snr_db=20.0, seed=4, n_targets=3, extent=3.0)
    want = O.range_compress_fp64(sc.phase_history, sc.nfft, O.hamming(K))
    with focusing.Plan.for_scene(sc, "mixed") as plan:
        assert plan.info["fused_range_compression"] == 1
        for n in (1, 5):
            plan.range_compress(np.ascontiguousarray(sc.phase_history[:n]))
            assert O.rel_l2(plan.range_profiles(), want[:n]) < 2e-6


@pytest.mark.parametrize("K,R,cap,chirp", [(272, 4, 768, 1), (272, 4, 769, 0), (372, 8, 1000, 0), (380, 8, 768, 1),
                                           (399, 8, 2048, 1), (319, 4, 2048, 1), (377, 8, 2048, 1), (296, 4, 2048, 1),
                                           (260, 4, 64, 0), (512, 8, 2048, 0)])
def test_chirp_rule(K, R, cap, chirp):
    """Either side of the rule's lines: by the number of pulses where the
    longest factor is 17 to 31, by the factors elsewhere."""
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from uncc_sar_focusing_b200 import focusing

    sc = S.point_target_scene(K=K, Np=7, n=16, spacing=0.2, nfft=R * K, snr_db=20.0, seed=4, n_targets=3, extent=3.0)
    want = O.range_compress_fp64(sc.phase_history, sc.nfft, O.hamming(K))
    with focusing.Plan(K, cap, R * K, sc.max_wr, sc.grid) as plan:
        assert plan.info["chirp_range_compression"] == chirp
        plan.range_compress(sc.phase_history)
        assert O.rel_l2(plan.range_profiles(), want) < 2e-6
