"""Routes that meet only in a batch or a hypothesis launch, against the FP64
oracle's 1e-4 relative L2: chirp, direct and cuFFT range compression side by
side, more scenes of one shape than a range-compression launch holds, tiles taken
with rows and columns exchanged beside tiles that are not."""
import numpy as np
import pytest

from oracle import oracle as O
from uncc_sar_focusing_b200 import scenes as S

pytestmark = pytest.mark.gpu
TOL = 1e-4


@pytest.fixture(scope="module")
def F():
    import torch

    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from uncc_sar_focusing_b200 import focusing

    return focusing


def scene(K, R, Np, nx, ny, seed, side):
    """side: seen from the y axis (64-row tiles are exchanged)."""
    sc = S.point_target_scene(K=K, Np=Np, n=40, spacing=0.1, nfft=R * K, snr_db=20.0, seed=seed, n_targets=4, extent=3.0)
    sc.grid = S.Grid(nx=nx, ny=ny, wx=0.1 * (nx - 1), wy=0.12 * (ny - 1), x0=0.4, y0=-0.3)
    if side:
        sc.ant_x, sc.ant_y = sc.ant_y, sc.ant_x
    return sc


def args(sc):
    import torch

    return tuple(torch.as_tensor(np.ascontiguousarray(a)).cuda()
                 for a in (sc.phase_history, sc.ant_x, sc.ant_y, sc.ant_z, sc.slant_range, sc.start_freq))


@pytest.mark.parametrize("per_tile", [False, True])
def test_mixed_routes(F, per_tile):
    shapes = [(424, 8, 40), (501, 4, 21), (256, 4, 33), (40, 6, 17), (424, 8, 25), (512, 8, 30), (280, 8, 12)]
    scs = [scene(K, R, n, 64 + 61 * (i % 2), 70 + 9 * i, i, i % 3 != 0) for i, (K, R, n) in enumerate(shapes)]
    with F.Batch(scs) as batch:
        assert batch.info["tile_mx"] == 8  # the tiles that can be exchanged
        batch.set_schedule(per_tile)
        imgs = batch.new_images()
        for _ in range(2):  # captured, then replayed
            batch.focus([args(sc) for sc in scs], imgs)
            batch.wait()
    for sc, img in zip(scs, imgs):
        assert O.rel_l2(img.cpu().numpy(), O.focus_fp64(sc)) < TOL


@pytest.mark.parametrize("K,R", [(256, 2), (424, 4)])
def test_more_scenes_of_one_shape_than_a_launch_holds(F, K, R):
    scs = [scene(K, R, 3 + i % 4, 9 + i % 5, 11, i, i % 2 == 1) for i in range(70)]
    with F.Batch(scs) as batch:
        imgs = batch.new_images()
        batch.focus([args(sc) for sc in scs], imgs)
        batch.wait()
    for sc, img in zip(scs, imgs):
        assert O.rel_l2(img.cpu().numpy(), O.focus_fp64(sc)) < TOL


@pytest.mark.parametrize("nx,ny,Np", [(64, 64, 40), (124, 70, 37)])
def test_hypotheses_from_two_sides(F, nx, ny, Np):
    tracks = [scene(64, 8, Np, nx, ny, 2, side) for side in (False, True, True, False, True)]
    geo = [np.stack([getattr(t, k) for t in tracks]) for k in ("ant_x", "ant_y", "ant_z", "slant_range", "start_freq")]
    with F.Plan.for_scene(tracks[0], "mixed") as plan:
        assert plan.info["tile_mx"] == 8
        plan.range_compress(tracks[0].phase_history)
        got = plan.backproject_hypotheses(*geo)
    for t, img in zip(tracks, got):
        assert O.rel_l2(img, O.focus_fp64(t)) < TOL
