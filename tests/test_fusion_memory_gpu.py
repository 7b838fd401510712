"""Fusion on a device that runs out of memory: what it can do without goes first."""
import numpy as np
import pytest

from sensemap_b200 import _native as N
from sensemap_b200 import synthetic as syn
from sensemap_b200.fusion import FusionOptions, StereoFusion

pytestmark = pytest.mark.gpu


def _inputs():
    scene = syn.heightfield_scene(seed=9, width=96, height=72, focal=72.0, num_src=3, device="cuda")
    return syn.fusion_inputs(scene, seed=3)


def _fuse(images, overlaps, fail_at):
    """The points, or None where the call reported that memory ran out."""
    lib = N.lib()
    N.check(lib.smvs_test_fail_allocation(fail_at))
    try:
        with StereoFusion(FusionOptions(), images, overlaps) as f:
            f.Run()
            return f.GetFusedPoints().copy()
    except N.SmvsError as error:
        assert error.status == N.SMVS_ENOMEM
        return None
    finally:
        N.check(lib.smvs_test_fail_allocation(0))


@pytest.mark.parametrize("in_place", [0, 1])
def test_any_allocation_may_fail(in_place):
    """The nth allocation fails, for every n. Once the projection table is there it
    makes room for whatever comes after; without one, the predecessor lists can be
    left out. No failure changes the points."""
    images, overlaps = _inputs()
    want = _fuse(images, overlaps, 0)
    assert len(want) > 100
    N.check(N.lib().smvs_test_fusion_paths(in_place, 0))
    try:
        failed, total = [], 70
        for nth in range(1, total + 1):
            got = _fuse(images, overlaps, nth)
            if got is None:
                failed.append(nth)
            else:
                np.testing.assert_array_equal(got.view(np.uint8), want.view(np.uint8))
    finally:
        N.check(N.lib().smvs_test_fusion_paths(0, 0))
    before_table = 21  # the arrays of all pixels and the record pool
    if in_place:
        assert max(failed) > before_table + 1 and max(failed) < total
        assert any(nth not in failed for nth in range(before_table + 1, max(failed)))
    else:
        assert failed == list(range(1, len(failed) + 1)) and len(failed) <= before_table


def test_overlap_list_of_an_unused_image_costs_nothing():
    """An image without a depth map overlaps all others many times over; the table's
    rows keep the width of the longest list of a used image."""
    images, overlaps = _inputs()
    want = _fuse(images, overlaps, 0)
    images = list(images) + [type(images[0])(K=images[0].K, R=images[0].R, T=images[0].T)]
    overlaps = list(overlaps) + [list(range(len(overlaps))) * 200]
    got = _fuse(images, overlaps, 0)
    np.testing.assert_array_equal(got.view(np.uint8), want.view(np.uint8))


@pytest.mark.parametrize("call", ["RemoveOutliers", "RemoveDuplicatePoints"])
def test_clean_up_can_be_called_again_after_it_ran_out_of_memory(call):
    """Two images from one place: a point for nearly every pixel pair, so that the
    clean-up does not fit into the image loop's arrays. Whichever allocation fails,
    the pass can be called again."""
    images, _ = _inputs()
    options = FusionOptions(min_num_pixels=2, max_num_pixels=2, min_num_visible_images=1, max_normal_error=90.0,
                            max_depth_error=0.1)
    keep = [images[0], images[0]]
    lists = [[1], [0]]

    def fusion():  # without the projection table, which would make room
        N.check(N.lib().smvs_test_fusion_paths(1, 0))
        try:
            return StereoFusion(options, keep, lists)
        finally:
            N.check(N.lib().smvs_test_fusion_paths(0, 0))

    with fusion() as f:
        f.Run()
        assert len(f.GetFusedPoints()) > 3 * keep[0].depth.size // 4
        points = len(f.GetFusedPoints())
    failures = 0
    for nth in range(1, 16):
        with fusion() as f:
            f.Run()
            N.check(N.lib().smvs_test_fail_allocation(nth))
            try:
                got = getattr(f, call)()
            except N.SmvsError as error:
                assert error.status == N.SMVS_ENOMEM
                got = None
            finally:
                N.check(N.lib().smvs_test_fail_allocation(0))
            if got is None:
                failures += 1
                got = getattr(f, call)()
            assert got <= points and len(f.GetFusedPoints()) == points - got
    assert failures < 15 and (failures > 0 or call == "RemoveDuplicatePoints")


@pytest.mark.parametrize("call", ["RemoveOutliers", "RemoveDuplicatePoints"])
def test_clean_up_that_runs_out_of_memory_leaves_the_cloud(call):
    """Two images from one place: a point for nearly every pixel pair, so that the
    clean-up does not fit into the image loop's arrays. Whichever allocation fails,
    points, scores and images stay as they were, and the next call gives what the
    first would have."""
    images, _ = _inputs()
    options = FusionOptions(min_num_pixels=2, max_num_pixels=2, min_num_visible_images=1, max_normal_error=90.0,
                            max_depth_error=0.1)
    keep = [images[0], images[0]]
    lists = [[1], [0]]

    def cloud(f):
        return [a.copy().view(np.uint8) for a in (f.GetFusedPoints(), *f.VisibilityCSR())]

    def same(a, b):
        for x, y in zip(a, b):
            np.testing.assert_array_equal(x, y)

    def fusion():  # without the projection table, which would make room
        N.check(N.lib().smvs_test_fusion_paths(1, 0))
        try:
            return StereoFusion(options, keep, lists)
        finally:
            N.check(N.lib().smvs_test_fusion_paths(0, 0))

    with fusion() as f:
        f.Run()
        assert len(f.GetFusedPoints()) > 3 * keep[0].depth.size // 4
        before = cloud(f)
        dropped = getattr(f, call)()
        after = cloud(f)
    failures = 0
    for nth in range(1, 16):
        with fusion() as f:
            f.Run()
            N.check(N.lib().smvs_test_fail_allocation(nth))
            try:
                got = getattr(f, call)()
            except N.SmvsError as error:
                assert error.status == N.SMVS_ENOMEM
                got = None
            finally:
                N.check(N.lib().smvs_test_fail_allocation(0))
            if got is None:
                failures += 1
                same(cloud(f), before)
                got = getattr(f, call)()
            assert got == dropped
            same(cloud(f), after)
    assert failures < 15 and (failures > 0 or call == "RemoveDuplicatePoints")
