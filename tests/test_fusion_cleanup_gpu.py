"""GPU parity of the fusion clean-up passes against the C oracle.

The fused cloud of the GPU image loop is cleaned on the GPU
(smvs_fusion_remove_duplicate_points, smvs_fusion_remove_outliers) and, from
the same cloud, by the oracle (oracle/smvs_oracle_fusion.c: the greedy
duplicate loop of RemoveDuplicatePoints and RemoveOutliers with brute-force
neighbours). Kept points (every field, bit for bit, scores included), their
images and the counts dropped must be identical.
"""
import numpy as np
import pytest

from oracle import oracle as O
from sensemap_b200 import synthetic as syn
from sensemap_b200.fusion import FusionOptions, StereoFusion

pytestmark = pytest.mark.gpu


def _cloud(f):
    pts = f.GetFusedPoints().copy()
    off, vis = f.VisibilityCSR()
    return pts, off.copy(), vis.copy()


def _same_cloud(a, b):
    assert len(a[0]) == len(b[0]), (len(a[0]), len(b[0]))
    assert np.array_equal(a[0].view(np.uint8), b[0].view(np.uint8))
    assert np.array_equal(a[1], b[1])
    assert np.array_equal(a[2], b[2])


@pytest.mark.parametrize("scene_kind", ["planes", "heightfield"])
def test_cleanup_matches_oracle(scene_kind):
    if scene_kind == "planes":
        scene = syn.planes_scene(seed=3, width=200, height=150, focal=160.0, num_src=4)
    else:
        scene = syn.heightfield_scene(seed=2, width=320, height=240, focal=240.0, num_src=5)
    ims, ov = syn.fusion_inputs(scene, seed=1)
    with StereoFusion(FusionOptions(), ims, ov) as f:
        f.Run()
        fused = _cloud(f)
        dropped = f.RemoveDuplicatePoints()
        dedup = _cloud(f)
        kp, ko, kv, o_dropped = O.fusion_remove_duplicates(ims, *fused)
        assert dropped == o_dropped
        _same_cloud(dedup, (kp, ko, kv))
        removed = f.RemoveOutliers(nb_neighbors=6, max_spacing_factor=6.0)
        clean = _cloud(f)
        rp, ro, rv, o_removed, _ = O.fusion_remove_outliers(*dedup, nb_neighbors=6, max_spacing_factor=6.0)
        assert removed == o_removed
        _same_cloud(clean, (rp, ro, rv))
    assert len(fused[0]) > 500


def test_outlier_pass_with_far_points_and_other_neighbour_counts():
    scene = syn.planes_scene(seed=5, width=160, height=120, focal=128.0, num_src=4)
    ims, ov = syn.fusion_inputs(scene, seed=3)
    for nb in (1, 12):
        with StereoFusion(FusionOptions(), ims, ov) as f:
            f.Run()
            before = _cloud(f)
            removed = f.RemoveOutliers(nb_neighbors=nb, max_spacing_factor=3.0)
            after = _cloud(f)
        rp, ro, rv, o_removed, _ = O.fusion_remove_outliers(*before, nb_neighbors=nb, max_spacing_factor=3.0)
        assert removed == o_removed
        _same_cloud(after, (rp, ro, rv))


@pytest.mark.parametrize("nb", [1, 7, 8, 15, 16, 63])
def test_cleanup_of_scattered_points(nb):
    """Loose fusion of noisy maps: points that stand alone (their neighbours lie many
    cells away), every number of images, and each form of the neighbour search at the
    ends of its range. The passes come in both orders and twice."""
    scene = syn.heightfield_scene(seed=6, width=96, height=72, focal=72.0, num_src=5)
    ims, ov = syn.fusion_inputs(scene, seed=4)
    rng = np.random.default_rng(nb)
    for im in ims:
        hit = rng.random(im.depth.shape) < 0.1
        im.depth[hit] *= rng.choice([0.3, 0.7, 1.6, 5.0], int(hit.sum())).astype(np.float32)
    opt = FusionOptions(min_num_pixels=2, min_num_visible_images=2, max_normal_error=60.0, max_depth_error=0.05)
    with StereoFusion(opt, ims, ov) as f:
        f.Run()
        cloud = _cloud(f)
        assert len(cloud[0]) > 200
        for k in range(4):
            if k % 2 == 0:
                removed = f.RemoveOutliers(nb_neighbors=nb, max_spacing_factor=2.0)
                p, o, v, want, _ = O.fusion_remove_outliers(*cloud, nb_neighbors=nb, max_spacing_factor=2.0)
            else:
                removed = f.RemoveDuplicatePoints()
                p, o, v, want = O.fusion_remove_duplicates(ims, *cloud)
            assert removed == want
            cloud = _cloud(f)
            _same_cloud(cloud, (p, o, v))


def test_cleanup_of_an_empty_cloud():
    scene = syn.planes_scene(seed=3, width=40, height=30, focal=32.0, num_src=2)
    ims, ov = syn.fusion_inputs(scene, seed=1)
    with StereoFusion(FusionOptions(min_num_pixels=10000), ims, ov) as f:
        f.Run()
        assert f.RemoveDuplicatePoints() == 0 and f.RemoveOutliers() == 0
        assert len(f.GetFusedPoints()) == 0
